// neighbor.cu -- Verlet list (cutoff + skin) on a cell grid; the per-step
// typewise radial / angular filter of its rows is k_filter_radial
// (nep_force.cu).
//
// Reference behaviour (src/gpumd_compat/neighbor.cu:90-582, nep.cu:503-561):
// the Verlet list of all pairs with float d^2 < (rc + skin)^2 is rebuilt when
// any atom moved more than skin/2 since the last build; every force call
// filters it into typewise radial and angular lists with float
// d^2 < ((rc_t1 + rc_t2)/2)^2.  Rows are ascending in atom index.
//
// B200 design: everything stays on the device.  The skin check is a plain kernel
// (in an MD step, part of the first half kick); the rebuild is one cooperative
// launch whose phases -- cell grid, counting sort of the atoms into cells, Verlet
// rows -- are separated by grid-wide barriers (every block is resident, and every
// wait is bounded).  A step with nothing to rebuild costs that launch, which
// returns at once, and never waits on the host.  Rows are row-major (atom i owns the contiguous
// slots [i*MN, i*MN + count)) so the warp that owns a center reads and writes
// coalesced.  The cell list is a counting sort on a grid of cells at least
// (rc + skin)/2 wide with a 5x5x5 stencil; each Verlet row is sorted (in
// registers, above 256 entries in shared memory), which makes every later sum over
// neighbours ordered and bitwise reproducible.
#include <algorithm>
#include <climits>

#include "engine.h"
#include "stencil.cuh"

namespace nepx {

namespace {

// Sixteen warps, a center per warp in the row build: CTAs of four warps hold the
// same number, but four times the arrivals at every barrier.
constexpr int kRebuildThreads = 512;
constexpr int kRebuildCtas = 3;                      // per SM (40 registers, the most for three; 72 bytes spilled)
constexpr int kRebuildWarps = kRebuildThreads / 32;
constexpr long long kGridWaitCycles = 4000000000ll;  // ~2 s at the B200 clock

__device__ __forceinline__ int wrapped_cell(double s, int nc, int pbc)
{
  if (!pbc) return 0;
  s -= floor(s);
  int c = static_cast<int>(s * nc);
  return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

// Packs each atom into its Site record for the neighbour sweeps of this
// step and applies the skin criterion (skin_check_atom, common.cuh); the MD
// step does the same inside its first half kick instead.  The call's box, when it
// brings one, goes to the device copy here.  (As the first phase of the
// cooperative rebuild it put a grid-wide barrier on every call: neighbour stage
// of 24,000 atoms 19 us, of 1,551 atoms 11 us.)
__global__ void __launch_bounds__(256)
k_skin(int N, Box* box, int set_box, const Box host_box, const double* __restrict__ pos,
       const int* __restrict__ type, const double* __restrict__ x0, NeighborState* st,
       Site* __restrict__ sites, double skin, double rc_v, int force)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (set_box && i == 0) *box = host_box;   // for the launches that follow
  if (i >= N) return;
  const Box* b = box;
  Box mine;
  if (set_box) mine = host_box;
  else mine = *b;
  skin_check_atom(N, i, mine, pos[i], pos[N + i], pos[2 * N + i], type[i], x0, st, sites, skin,
                  rc_v, force);
}

// Grid-wide barrier of the cooperative rebuild.  A generation counter: the
// last block to arrive resets the arrival count and advances the generation,
// the others wait for the advance -- at most kGridWaitCycles, after which they
// record the timeout in sync_error and go on (the call then reports an error).
__device__ void grid_sync(unsigned* gs, NeighborState* st)
{
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* gen = gs + 1;
    const unsigned g = *gen;
    __threadfence();
    if (atomicAdd(gs, 1u) == gridDim.x - 1) {
      atomicExch(gs, 0u);
      __threadfence();
      atomicAdd(gs + 1, 1u);
    } else {
      const long long t0 = clock64();
      while (*gen == g) {
        if (clock64() - t0 > kGridWaitCycles) {
          atomicOr(&st->sync_error, 1);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// Sum over the block (kRebuildThreads threads).
__device__ int block_sum(int v, int* s_tmp)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) s_tmp[warp] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < kRebuildWarps; ++w) t += s_tmp[w];
  return t;
}

// Inclusive prefix sum over the block; *total gets the block's sum.
__device__ int block_scan(int v, int* s_tmp, int* total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) s_tmp[warp] = x;
  __syncthreads();
  int before = 0, t = 0;
  for (int w = 0; w < kRebuildWarps; ++w) {
    if (w < warp) before += s_tmp[w];
    t += s_tmp[w];
  }
  *total = t;
  return x + before;
}

// Compare-exchange of two values held by one lane: the pair's lower element
// keeps the smaller value when its block sorts ascending.
__device__ __forceinline__ void cx_pair(int& lo, int& hi, bool ascending)
{
  const int a = min(lo, hi), c = max(lo, hi);
  lo = ascending ? a : c;
  hi = ascending ? c : a;
}

// Ascending bitonic sort of the first p2 (a power of two, at most 32 R) values
// of a warp, R per lane: element e = lane + 32 r is v[r] (padding INT_MAX).
// Partners e ^ jj exchange by shuffle (jj < 32) or inside the lane (jj >= 32);
// e keeps the smaller value when (e < partner) matches the ascending direction
// (e & k) == 0 of its block.
template <int R>
__device__ __forceinline__ void warp_sort(int (&v)[R], int p2, int lane)
{
  for (int k = 2; k <= p2; k <<= 1) {
#pragma unroll
    for (int step = R / 2; step > 0; step >>= 1) {
      if (32 * step <= (k >> 1)) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if ((r & step) == 0) cx_pair(v[r], v[r + step], ((lane + 32 * r) & k) == 0);
      }
    }
    for (int jj = min(16, k >> 1); jj > 0; jj >>= 1) {
      const bool lower = (lane & jj) == 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int pv = __shfl_xor_sync(0xffffffffu, v[r], jj);
        const bool asc = ((lane + 32 * r) & k) == 0;
        v[r] = (lower == asc) ? min(v[r], pv) : max(v[r], pv);
      }
    }
  }
}

// Sorts the used first entries of buf in registers and writes keep of them.
template <int R>
__device__ __forceinline__ void sort_row(const int* buf, int used, int p2, int keep, int* row,
                                         int lane)
{
  int v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = lane + 32 * r < used ? buf[lane + 32 * r] : INT_MAX;
  warp_sort(v, p2, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane + 32 * r < keep) row[lane + 32 * r] = v[r];
}

struct RebuildArgs {
  int N;
  const Box* box;
  const double* pos;
  const int* type;
  NeighborState* st;
  Site* sites;
  int* cell_count;
  int* cell_start;
  int* cell_atoms;
  int* cell_of;
  Site* cell_sites;    // the site records in cell order (beside cell_atoms)
  int* nn_v;
  int* nl_v;
  double* x0;
  unsigned* gsync;
  int* part;           // [gridDim.x] per-block sums of the cell scan
  int mn_v, pow2, cell_cap;
  double rc_v;
  float cutoff_square;
  double prune_square; // (rc_v (1 + 1e-5) + 1e-5)^2: the stencil rows' trimming bound
};

// The rebuild of the Verlet rows in one cooperative launch (grid-stride phases,
// grid_sync between them), after the site records and the skin criterion:
//   1. cell grid from the current box (cells at least rc_v/2 thick, at most
//      cell_cap of them), counts cleared;
//   2. cell of every atom, counts;
//   3. exclusive scan of the counts (per-block chunks, then block offsets);
//   4. atoms into their cells (index and site record, in cell order);
//   5. Verlet rows: one warp per center gathers every candidate of the 5x5x5
//      stencil (its rows along x, trimmed to the cells in reach) with float
//      d^2 < (rc + skin)^2, sorts the row (bitonic, in registers up to 256
//      entries) and writes it with the reference positions of the next skin
//      check.
// They run only when the rebuild flag is set; the flag is the same for every
// block, so all of them return together.
__global__ void __launch_bounds__(kRebuildThreads, kRebuildCtas)
k_neighbor_rebuild(const RebuildArgs a)
{
  extern __shared__ int s_rows[];
  __shared__ int s_tmp[kRebuildWarps];
  __shared__ int s_grid[4];
  NeighborState* st = a.st;
  const int N = a.N;
  const int tid = threadIdx.x;
  const int gtid = blockIdx.x * blockDim.x + tid, nthreads = gridDim.x * blockDim.x;
  if (!st->rebuild) return;
  const Box b = *a.box;

  // 1. cell grid (every block derives the same one; block 0 records it)
  if (tid == 0) {
    int nc[3];
    double width = 0.5 * a.rc_v;
    for (int pass = 0; pass < 64; ++pass) {
      long long total = 1;
      for (int d = 0; d < 3; ++d) {
        // thickness along direction d = 1 / |row d of hinv|
        const double* r = b.hinv + 3 * d;
        const double thick = 1.0 / sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
        nc[d] = b.pbc[d] ? max(1, static_cast<int>(floor(thick / width))) : 1;
        total *= nc[d];
      }
      if (total <= a.cell_cap) break;
      width *= 1.25;
    }
    s_grid[0] = nc[0];
    s_grid[1] = nc[1];
    s_grid[2] = nc[2];
    s_grid[3] = nc[0] * nc[1] * nc[2];
    if (blockIdx.x == 0) {
      st->box_scale = 1.0;
      for (int k = 0; k < 9; ++k) st->box_def[k] = (k % 4 == 0) ? 1.0 : 0.0;
      st->nc[0] = nc[0];
      st->nc[1] = nc[1];
      st->nc[2] = nc[2];
      st->ncell = s_grid[3];
    }
  }
  __syncthreads();
  const int nc0 = s_grid[0], nc1 = s_grid[1], nc2 = s_grid[2], ncell = s_grid[3];
  for (int c = gtid; c < ncell; c += nthreads) a.cell_count[c] = 0;
  grid_sync(a.gsync, st);

  // 2. cells and counts
  for (int i = gtid; i < N; i += nthreads) {
    const double x = a.pos[i], y = a.pos[N + i], z = a.pos[2 * N + i];
    const double sx = b.hinv[0] * x + b.hinv[1] * y + b.hinv[2] * z;
    const double sy = b.hinv[3] * x + b.hinv[4] * y + b.hinv[5] * z;
    const double sz = b.hinv[6] * x + b.hinv[7] * y + b.hinv[8] * z;
    const int c = (wrapped_cell(sz, nc2, b.pbc[2]) * nc1 + wrapped_cell(sy, nc1, b.pbc[1])) * nc0 +
                  wrapped_cell(sx, nc0, b.pbc[0]);
    a.cell_of[i] = c;
    atomicAdd(a.cell_count + c, 1);
  }
  grid_sync(a.gsync, st);

  // 3. exclusive scan: block sums of contiguous chunks, then each block
  //    scans its chunk from the sum of the chunks before it; the counts
  //    are reset to serve as fill cursors
  const int chunk = (ncell + gridDim.x - 1) / gridDim.x;
  const int c0 = min(ncell, static_cast<int>(blockIdx.x) * chunk), c1 = min(ncell, c0 + chunk);
  {
    int sum = 0;
    for (int c = c0 + tid; c < c1; c += blockDim.x) sum += a.cell_count[c];
    sum = block_sum(sum, s_tmp);
    if (tid == 0) a.part[blockIdx.x] = sum;
  }
  grid_sync(a.gsync, st);
  {
    int off = 0;
    for (int q = tid; q < static_cast<int>(blockIdx.x); q += blockDim.x) off += a.part[q];
    off = block_sum(off, s_tmp);
    for (int base = c0; base < c1; base += blockDim.x) {
      const int c = base + tid;
      const int v = c < c1 ? a.cell_count[c] : 0;
      int tile = 0;
      const int incl = block_scan(v, s_tmp, &tile);
      if (c < c1) {
        a.cell_start[c] = off + incl - v;
        a.cell_count[c] = 0;
      }
      off += tile;
    }
  }
  grid_sync(a.gsync, st);

  // 4. fill (the counts are the cell totals again afterwards); each atom's
  //    site record goes beside its index, so a cell's candidates are one
  //    contiguous run of records
  for (int i = gtid; i < N; i += nthreads) {
    const int c = a.cell_of[i];
    const int slot = atomicAdd(a.cell_count + c, 1);
    const int at = a.cell_start[c] + slot;
    a.cell_atoms[at] = i;
    a.cell_sites[at] = a.sites[i];
  }
  grid_sync(a.gsync, st);

  // 5. Verlet rows, one warp per center (stencil.cuh); each candidate's index
  //    and site record are read side by side.  Hits are compacted in order of
  //    discovery (ballot + popcount) and the row is sorted: in registers up to
  //    256 entries, in shared memory above.
  const int lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int pow2 = a.pow2;
  int* buf = s_rows + warp * (pow2 + 1);
  const CellGrid grid{{nc0, nc1, nc2}, {b.h[0] / nc0, b.h[4] / nc1, b.h[8] / nc2}, 0};
  for (int i = blockIdx.x * kRebuildWarps + warp; i < N; i += gridDim.x * kRebuildWarps) {
    const double xi = a.sites[i].x, yi = a.sites[i].y, zi = a.sites[i].z;
    const Stencil cand(b, grid, a.cell_of[i], xi, yi, zi, a.prune_square, a.cell_start,
                       a.cell_count, lane);
    int total = 0;
    for (int base = 0; base < cand.total; base += 32) {
      const int k = base + lane;
      const int at = cand.place(k);
      bool hit = false;
      int j = 0;
      if (k < cand.total) {
        j = a.cell_atoms[at];
        double2 sa, sc;
        site_load_coherent(a.cell_sites, at, sa, sc);
        float dx, dy, dz;
        int tj;
        site_delta(b, sa, sc, xi, yi, zi, dx, dy, dz, tj);
        const float d2 = dx * dx + dy * dy + dz * dz;
        hit = j != i && d2 < a.cutoff_square;
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int slot = total + __popc(m & below);
        if (slot < pow2) buf[slot] = j;
      }
      total += __popc(m);
    }
    __syncwarp();
    const int used = min(total, pow2);
    int p2 = 1;
    while (p2 < used) p2 <<= 1;
    const int keep = min(total, a.mn_v);
    int* row = a.nl_v + static_cast<size_t>(i) * a.mn_v;
    if (p2 <= 128) {
      sort_row<4>(buf, used, p2, keep, row, lane);
    } else if (p2 == 256) {
      // (in shared memory: 36 passes of four pairs per lane; the rebuild of 24,000
      // water atoms, whose rows hold 144, 271 -> 171 us)
      sort_row<8>(buf, used, p2, keep, row, lane);
    } else {
      // bitonic sort of the smallest power of two that holds the row (padding
      // INT_MAX), one compare-exchange pair per lane and pass
      for (int k = used + lane; k < p2; k += 32) buf[k] = INT_MAX;
      __syncwarp();
      for (int k = 2; k <= p2; k <<= 1) {
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
          for (int q = lane; q < (p2 >> 1); q += 32) {
            const int t = ((q & ~(jj - 1)) << 1) | (q & (jj - 1));   // lower index of the pair
            const int u = t | jj;
            const int x = buf[t], y = buf[u];
            const bool up = (t & k) == 0;
            if ((x > y) == up) {
              buf[t] = y;
              buf[u] = x;
            }
          }
          __syncwarp();
        }
      }
      for (int k = lane; k < keep; k += 32) row[k] = buf[k];
    }
    if (lane == 0) {
      a.nn_v[i] = keep;
      if (total > a.mn_v) atomicOr(&st->overflow, 1);
      atomicMax(&st->max_nn[0], total);
      a.x0[i] = xi;
      a.x0[N + i] = yi;
      a.x0[2 * N + i] = zi;
    }
    __syncwarp();   // the row buffer is reused by this warp's next center
  }
}

size_t rebuild_smem(int pow2) { return sizeof(int) * kRebuildWarps * (pow2 + 1); }

}  // namespace

// Blocks of the cooperative rebuild: as many as can be resident at once (the
// launch fails rather than oversubscribe): three per SM, fewer for long rows' sort
// buffers.
int neighbor_rebuild_blocks(int pow2_v)
{
  int dev = 0, sms = 0, per_sm = 0;
  // long rows' sort buffers exceed the default limit (rows are capped at 2,048)
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaFuncSetAttribute(k_neighbor_rebuild, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(rebuild_smem(2048))) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_neighbor_rebuild, kRebuildThreads,
                                                    rebuild_smem(pow2_v)) != cudaSuccess)
    return 0;
  return sms * per_sm;
}

void launch_neighbor_update(Engine& e, int N, const double* pos, const int* type, bool force,
                            cudaStream_t stream, bool skin_done)
{
  if (e.use_xr) {
    launch_explicit_rows(e, N, pos, type, stream);
    return;
  }
  NeighborBuffers& nb = e.nbr;
  if (nb.gsync_dirty) {
    // a barrier gave up waiting in an earlier launch: restart its counters
    cudaMemsetAsync(nb.gsync, 0, 2 * sizeof(unsigned), stream);
    nb.gsync_dirty = false;
  }
  RebuildArgs a;
  a.N = N;
  a.box = e.d_box;
  a.pos = pos;
  a.type = type;
  a.st = e.d_nstate;
  a.sites = e.scratch.sites;
  a.cell_count = nb.cell_count;
  a.cell_start = nb.cell_start;
  a.cell_atoms = nb.cell_atoms;
  a.cell_of = nb.cell_of;
  a.cell_sites = nb.cell_sites;
  a.nn_v = nb.nn_v;
  a.nl_v = nb.nl_v;
  a.x0 = nb.x0;
  a.gsync = nb.gsync;
  a.part = nb.scan_part;
  a.mn_v = nb.mn_v;
  a.pow2 = nb.pow2_v;
  a.cell_cap = nb.cell_cap;
  a.rc_v = static_cast<double>(e.model.rc_max) + e.skin;
  a.cutoff_square = static_cast<float>(a.rc_v * a.rc_v);
  const double rp = a.rc_v * (1.0 + 1e-5) + 1e-5;
  a.prune_square = rp * rp;
  if (!skin_done)
    k_skin<<<(N + 255) / 256, 256, 0, stream>>>(N, e.d_box, e.staged_box ? 1 : 0,
                                                e.staged_box ? *e.staged_box : Box{}, pos, type,
                                                nb.x0, e.d_nstate, e.scratch.sites, e.skin, a.rc_v,
                                                force ? 1 : 0);
  // small systems take fewer blocks: cheaper barriers, nothing to share out
  const int want = std::max(1, (N + kRebuildWarps - 1) / kRebuildWarps);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(std::min(nb.rebuild_blocks, want)));
  cfg.blockDim = dim3(kRebuildThreads);
  cfg.dynamicSmemBytes = rebuild_smem(nb.pow2_v);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_neighbor_rebuild, a);
  // the typewise radial / angular filter follows in k_filter_radial (which
  // clears the rebuild flag)
}

}  // namespace nepx
