// common.cuh -- shared device-side definitions of the nepx engine.
//
// Box and minimum image, NEP constants, cutoff and Chebyshev radial basis,
// and the real solid harmonics used by the descriptor and force kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nepx {

constexpr int kMaxTypes = 16;
constexpr int kMaxBasis = 17;   // basis_size + 1
constexpr int kMaxN = 13;       // n_max + 1
constexpr int kNumLM = 24;      // (L_max + 1)^2 - 1 at L_max = 4
constexpr int kNumLMHigh = 80;  // (L_max + 1)^2 - 1 at L_max = 8, the largest the format has
constexpr int kMaxDim = 128;
constexpr int kMaxInv = 6;      // q_222, q_1111, q_112, q_123, q_233, q_134
constexpr double kBoltzmann = 8.617343e-5;           // eV/K, GPUMD natural units
constexpr double kTimeUnit = 1.018051e+1;            // natural time unit in fs
constexpr double kPressureUnit = 1.602177e+2;        // eV/A^3 in GPa
constexpr float kCoulomb = 14.399645f;               // e^2/(4 pi eps0) in eV A

// Device-resident periodic box.  h is row-major with the cell vectors a, b, c
// as columns (the layout of the reference's Box::cpu_h[0..8]); hinv its
// inverse; fh the float copy (h then hinv) the FP32 kernels use.
struct Box {
  double h[9];
  double hinv[9];
  float fh[18];
  int pbc[3];
  int ortho;
};

// One structure of an explicit-row evaluation (the small-box path, and every
// structure of a batch): its box, the reference's expanded box for the image
// arithmetic, and its slice [off, off + n) of the concatenated atom arrays.
struct StructInfo {
  Box box;
  float eh[18];   // expanded box h (columns scaled by ncell) then its float inverse
  int ncell[3];   // images per direction (1 where not periodic)
  int small;      // 1: the reference's small-box image arithmetic; 0: minimum image
  int off, n;
  int nc[3];      // cell grid of a large structure's candidate search (nc[0] = 0: scan all atoms)
  int cell_base;  // first cell of this structure in the batch's cell arrays
  double cell_w[3];   // widths of the cells (orthogonal boxes)
  int keep;       // 1: keeps Verlet candidates across steps (cells sized for rc + skin)
};

// Packed neighbour of an explicit row: index j (low 28 bits) and type (high 4).
constexpr int kRowTypeShift = 28;
constexpr int kRowIndexMask = (1 << kRowTypeShift) - 1;

// Cell grid and rebuild bookkeeping of the Verlet list, device resident.
struct NeighborState {
  int rebuild;         // 1: rebuild the Verlet list before the next filter
  int overflow;        // bit 0 Verlet row, bit 1 radial row, bit 2 angular row
  int nc[3];           // cells per direction
  int ncell;
  int max_nn[3];       // largest Verlet / radial / angular row since the last stats read
  int call_nn[2];      // largest radial / angular row of the latest force evaluation
  int nonfinite;       // a force or energy came out NaN/Inf
  int box_error;       // the device box became unsupported (small in one direction, >10 rc in another)
  int ann_error;       // a tensor-core ANN tile gave up waiting for its MMAs
  int sync_error;      // the neighbour rebuild gave up waiting at a grid-wide barrier
  unsigned xr_builds;  // centers whose batch Verlet candidates were built (wraps)
  double box_scale;    // product of isotropic box factors since the last build (1 = none)
  double box_def[9];   // product of general box deformations since the last build (I = none)
};

// Minimum image of a float displacement, the arithmetic of the large-box
// path (reference box.cuh:84-127): half-box shortcut for orthogonal boxes,
// fractional nearbyint otherwise.
__device__ __forceinline__ void mic_f32(const Box& b, float& x, float& y, float& z)
{
  if (b.ortho) {
    const float lx2 = b.fh[0] * 0.5f, ly2 = b.fh[4] * 0.5f, lz2 = b.fh[8] * 0.5f;
    if (b.pbc[0] == 1) {
      if (x < -lx2) x += b.fh[0];
      else if (x > +lx2) x -= b.fh[0];
    }
    if (b.pbc[1] == 1) {
      if (y < -ly2) y += b.fh[4];
      else if (y > +ly2) y -= b.fh[4];
    }
    if (b.pbc[2] == 1) {
      if (z < -lz2) z += b.fh[8];
      else if (z > +lz2) z -= b.fh[8];
    }
  } else {
    float sx = b.fh[9] * x + b.fh[10] * y + b.fh[11] * z;
    float sy = b.fh[12] * x + b.fh[13] * y + b.fh[14] * z;
    float sz = b.fh[15] * x + b.fh[16] * y + b.fh[17] * z;
    if (b.pbc[0] == 1) sx -= nearbyintf(sx);
    if (b.pbc[1] == 1) sy -= nearbyintf(sy);
    if (b.pbc[2] == 1) sz -= nearbyintf(sz);
    x = b.fh[0] * sx + b.fh[1] * sy + b.fh[2] * sz;
    y = b.fh[3] * sx + b.fh[4] * sy + b.fh[5] * sz;
    z = b.fh[6] * sx + b.fh[7] * sy + b.fh[8] * sz;
  }
}

// The same minimum image with the box's numbers laid out for a sweep over
// neighbours: an orthogonal box's edges and half edges in registers, half an
// edge being infinite where the direction is not periodic (one comparison and
// one signed addition per direction, no test of the boundary); a general box's
// matrix and inverse in shared memory (18 floats), where they cost no registers.
// The results are mic_f32's bit for bit.
struct MinImage {
  float lx, ly, lz, hx, hy, hz;
  const float* fh;
  int pbc;
  bool ortho;

  // Called by every thread of the block, with a barrier before the first use;
  // s_fh: 18 floats of shared memory.
  __device__ __forceinline__ MinImage(const Box* __restrict__ b, float* s_fh)
    : MinImage(*b, static_cast<const float*>(s_fh))
  {
    for (int k = threadIdx.x; k < 18; k += blockDim.x) s_fh[k] = b->fh[k];
  }

  // The matrix read where it is (a warp with a box of its own).
  __device__ __forceinline__ explicit MinImage(const Box& b) : MinImage(b, b.fh) {}

  __device__ __forceinline__ MinImage(const Box& box, const float* matrix)
  {
    const Box* b = &box;
    fh = matrix;
    lx = b->fh[0];
    ly = b->fh[4];
    lz = b->fh[8];
    const float never = __int_as_float(0x7f800000);
    hx = b->pbc[0] == 1 ? lx * 0.5f : never;
    hy = b->pbc[1] == 1 ? ly * 0.5f : never;
    hz = b->pbc[2] == 1 ? lz * 0.5f : never;
    pbc = (b->pbc[0] == 1 ? 1 : 0) | (b->pbc[1] == 1 ? 2 : 0) | (b->pbc[2] == 1 ? 4 : 0);
    ortho = b->ortho != 0;
  }

  __device__ __forceinline__ void operator()(float& x, float& y, float& z) const
  {
    if (ortho) {
      if (fabsf(x) > hx) x -= copysignf(lx, x);
      if (fabsf(y) > hy) y -= copysignf(ly, y);
      if (fabsf(z) > hz) z -= copysignf(lz, z);
    } else {
      float sx = fh[9] * x + fh[10] * y + fh[11] * z;
      float sy = fh[12] * x + fh[13] * y + fh[14] * z;
      float sz = fh[15] * x + fh[16] * y + fh[17] * z;
      if (pbc & 1) sx -= nearbyintf(sx);
      if (pbc & 2) sy -= nearbyintf(sy);
      if (pbc & 4) sz -= nearbyintf(sz);
      x = fh[0] * sx + fh[1] * sy + fh[2] * sz;
      y = fh[3] * sx + fh[4] * sy + fh[5] * sz;
      z = fh[6] * sx + fh[7] * sy + fh[8] * sz;
    }
  }
};

// One atom as the neighbour sweeps read it: position and type in one
// 32-byte record (one sector), repacked from the SoA inputs at every force
// call.  The SoA layout would touch four cache lines per neighbour.
struct __align__(32) Site {
  double x, y, z;
  long long type;
};

// A site record in one 32-byte load: a = (x, y), c = (z, type bits).  Of 32
// scattered records in L1 the load pipe takes 26 cycles as two 16-byte loads
// each, 17.5 as one of 32 bytes, and the sweeps over neighbours are bound by it.
__device__ __forceinline__ void site_load(const Site* __restrict__ sites, int j, double2& a,
                                          double2& c)
{
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(a.x), "=d"(a.y), "=d"(c.x), "=d"(c.y)
      : "l"(sites + j));
}

// The same of a record that this launch may have written (coherent load).
__device__ __forceinline__ void site_load_coherent(const Site* sites, int j, double2& a,
                                                   double2& c)
{
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(a.x), "=d"(a.y), "=d"(c.x), "=d"(c.y)
               : "l"(sites + j)
               : "memory");
}

// Displacement from (xi, yi, zi) to a loaded site, and the site's type: the double
// difference rounded to float, then the float minimum image -- the operand order of
// the reference's filter (nep.cu:542-549), so neighbour predicates agree bit for bit.
__device__ __forceinline__ void site_delta(const Box& b, const double2& a, const double2& c,
                                           double xi, double yi, double zi, float& dx, float& dy,
                                           float& dz, int& tj)
{
  dx = a.x - xi;
  dy = a.y - yi;
  dz = c.x - zi;
  tj = static_cast<int>(__double_as_longlong(c.y));
  mic_f32(b, dx, dy, dz);
}

__device__ __forceinline__ void site_delta(const MinImage& mic, const double2& a, const double2& c,
                                           double xi, double yi, double zi, float& dx, float& dy,
                                           float& dz, int& tj)
{
  dx = a.x - xi;
  dy = a.y - yi;
  dz = c.x - zi;
  tj = static_cast<int>(__double_as_longlong(c.y));
  mic(dx, dy, dz);
}

// Skin criterion of atom i at its new position (reference
// neighbor.cu:446-533, without the host round trip): packs its Site record
// for this step's neighbour sweeps and marks a rebuild when forced or when
// it moved more than skin/2 since the build.  Under an isotropic box scaling
// s since the build (x0 scaled along, so displacements are co-moving) a pair
// distance also drifts by up to |1 - s| (rc + skin), which shrinks the
// allowed displacement to (skin - |1 - s| (rc + skin)) / 2.  A general
// deformation M since the build moves a pair by at most ||M - I||_2
// (rc + skin); the bound used is sqrt(||M - I||_1 ||M - I||_inf) >= ||M - I||_2.
__device__ __forceinline__ void skin_check_atom(int N, int i, const Box& b, double xi, double yi,
                                                double zi, int type_i,
                                                const double* __restrict__ x0, NeighborState* st,
                                                Site* __restrict__ sites, double skin,
                                                double rc_v, int force)
{
  sites[i] = Site{xi, yi, zi, static_cast<long long>(type_i)};
  if (i == 0) {   // the first kernel of a force evaluation: its row maxima start here
    st->call_nn[0] = 0;
    st->call_nn[1] = 0;
  }
  if (force) {
    if (i == 0) st->rebuild = 1;
    return;
  }
  double col[3] = {0.0, 0.0, 0.0}, row_max = 0.0;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    double row = 0.0;
    for (int c = 0; c < 3; ++c) {
      const double a = fabs(st->box_def[3 * r + c] - (r == c ? 1.0 : 0.0));
      row += a;
      col[c] += a;
    }
    row_max = fmax(row_max, row);
  }
  // (no deformation since the build, the usual case: no square root)
  const double def2 = fmax(fmax(col[0], col[1]), col[2]) * row_max;
  const double def = def2 == 0.0 ? 0.0 : sqrt(def2);
  const double strain = fmax(fabs(1.0 - st->box_scale), def);
  const double half = 0.5 * (skin - strain * rc_v);
  if (half <= 0.0) {
    st->rebuild = 1;
    return;
  }
  const double half_skin_sq = half * half;
  float dx = xi - x0[i];
  float dy = yi - x0[N + i];
  float dz = zi - x0[2 * N + i];
  mic_f32(b, dx, dy, dz);
  if ((dx * dx + dy * dy + dz * dz) > half_skin_sq) st->rebuild = 1;
}

// Two FP32 multiply-adds (or products) in one instruction: sm_100a's packed
// pairs, each half rounded as fmaf() rounds it.  The moment and force sweeps
// are bound by the instructions they issue, and half of those were FMAs.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
  float2 r;
  asm("{\n\t.reg .b64 a, b, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// Cutoff function fc = (1 + cos(pi d / rc)) / 2 and its d-derivative.
// On the one period's half that occurs, x = d / rc in [0, 1), both are short
// polynomials in t = x (1 - x) without a range reduction:
//   fc  = (1 - x) - y t S(t), y = x - 1/2: the cosine less its chord, which vanishes
//         with t. w = 1 - x is rounded below 1/2, and what it loses joins the
//         small term, so the sum is rounded once.
//   fc' = t R(t) / rc, since sin(pi x) is an entire function of t that vanishes with
//         it (so it keeps its relative accuracy at rc). R's constant -pi^2/2 is taken
//         in two parts, its leading product inside the last fma.
// S and R are least-maximum-error fits by iterated weighted least squares on
// Chebyshev nodes with the leading coefficients rounded first (residual 3e-9 and
// 1e-9).  Against 64 bits, over every float of [2^-10, 1) (in brackets the same
// from sincospif, which took some 30 instructions for the pair; these take about
// 18): fc at most 5.5e-8 (5.6e-8), rms 1.7e-8 (2.2e-8); fc' at most 1.2e-7 (1.7e-7)
// relative, rms 3.6e-8 (4.9e-8).  An earlier fit, fc = 1/2 - y P(y^2) without the
// chord, reached 8.1e-8 and 1.8e-7.
// FAST (the mixed-precision kernels): sine and cosine from the hardware
// approximations (absolute error about 4e-7 on [0, pi)).
template <bool FAST = false>
__device__ __forceinline__ void cutoff_fc(float rc, float rcinv, float d, float& fc, float& fcp)
{
  if (d < rc) {
    if constexpr (FAST) {
      float s, c;
      __sincosf(3.14159265f * (d * rcinv), &s, &c);
      fc = 0.5f * c + 0.5f;
      fcp = -1.5707963f * s * rcinv;
    } else {
      const float x = d * rcinv;
      const float t = fmaf(-x, x, x);
      float p = 0.0383364521f;
      p = fmaf(p, t, 0.260538638f);
      p = fmaf(p, t, 1.06520951f);
      p = fmaf(p, t, 2.0f);
      const float w = 1.0f - x;
      fc = w + fmaf((0.5f - x) * t, p, (1.0f - w) - x);
      float r = -0.0378732346f;
      r = fmaf(r, t, -0.321397096f);
      r = fmaf(r, t, -1.75220692f);
      r = fmaf(r, t, -4.93480158f);
      fcp = fmaf(t, -4.93480206f, t * fmaf(r, t, -1.45185794e-7f)) * rcinv;
    }
  } else {
    fc = 0.0f;
    fcp = 0.0f;
  }
}

// Edge length d and 1 / d from d^2: from one hardware reciprocal root y (2 ulp)
// by Markstein's method (P. W. Markstein, IBM J. Res. Dev. 34 (1990) 111), a Newton
// step of the root from d2 y and one of the reciprocal from y, each on a residual that
// an fma gives exactly.  7 instructions without a branch.  Over every float of two
// neighbouring binades d is sqrtf's and 1 / d within the error of the division
// (8.9e-8 against 64 bits, both).  FAST takes y itself.
template <bool FAST>
__device__ __forceinline__ void edge_length(float d2, float& d, float& dinv)
{
  if constexpr (FAST) {
    dinv = rsqrtf(d2);
    d = d2 * dinv;
  } else {
    const float y = rsqrtf(d2);
    const float d0 = d2 * y;
    d = fmaf(fmaf(-d0, d0, d2), 0.5f * y, d0);
    dinv = fmaf(fmaf(-d, y, 1.0f), y, y);
  }
}

// Functions past the model's basis multiply zero coefficients (the tables'
// rows are zero-padded), so a short basis is evaluated whole, without a
// comparison per function.
template <int KMAX>
__host__ __device__ constexpr bool whole_basis() { return KMAX <= 9; }

// Shifted Chebyshev radial basis f_k(d) = (T_k(x) + 1) / 2 * fc (f_0 = fc)
// with x = 2 (d/rc - 1)^2 - 1, k = 0..kmax-1.
template <int KMAX>
__device__ __forceinline__ void radial_basis(int kmax, float rcinv, float d, float fc, float* fn)
{
  const float u = d * rcinv - 1.0f;
  const float x = 2.0f * u * u - 1.0f;
  const float half_fc = 0.5f * fc, x2 = x + x;
  float t0 = 1.0f, t1 = x;
  fn[0] = fc;
#pragma unroll
  for (int k = 1; k < KMAX; ++k) {
    if (whole_basis<KMAX>() || k < kmax) fn[k] = fmaf(t1, half_fc, half_fc);
    const float t2 = fmaf(x2, t1, -t0);
    t0 = t1;
    t1 = t2;
  }
}

// Basis values and their d-derivatives,
// f'_k = T'_k (fc / 2) dx/dd + (T_k + 1) fc' / 2.
template <int KMAX>
__device__ __forceinline__ void radial_basis_d(int kmax, float rcinv, float d, float fc,
                                               float fcp, float* fn, float* fnp)
{
  const float u = d * rcinv - 1.0f;
  const float x = 2.0f * u * u - 1.0f;
  const float half_fc = 0.5f * fc, half_fcp = 0.5f * fcp, x2 = x + x;
  const float slope = half_fc * (4.0f * u * rcinv);   // (fc / 2) dx/dd
  float t0 = 1.0f, t1 = x;       // T_{k-1}, T_k
  float dt0 = 0.0f, dt1 = 1.0f;  // dT/dx
  fn[0] = fc;
  fnp[0] = fcp;
#pragma unroll
  for (int k = 1; k < KMAX; ++k) {
    if (whole_basis<KMAX>() || k < kmax) {
      fn[k] = fmaf(t1, half_fc, half_fc);
      fnp[k] = fmaf(dt1, slope, fmaf(t1, half_fcp, half_fcp));
    }
    const float t2 = fmaf(x2, t1, -t0);
    const float dt2 = fmaf(x2, dt1, fmaf(2.0f, t1, -dt0));
    t0 = t1;
    t1 = t2;
    dt0 = dt1;
    dt1 = dt2;
  }
}

// Real solid harmonics of degree L = 1..4 at the unit vector (x, y, z):
// Y = Z_Lm(z) * Re/Im (x + i y)^m with the z-polynomials below, in the
// component order of the reference's blm moments (L^2 - 1 + {0, 2m-1, 2m});
// zp[k] = z^k.  Degrees 5..8 read their coefficients from a table
// (harmonic_tables.h).
__device__ __forceinline__ float zpoly(int L, int m, const float* zp, float* dzf)
{
  // coefficients of the reference's Z_COEFFICIENT_L tables (nep_utilities.cuh:89-117)
  float f = 0.0f, df = 0.0f;
  switch (L * 8 + m) {
    case 8 + 0: f = zp[1]; df = 1.0f; break;
    case 8 + 1: f = 1.0f; df = 0.0f; break;
    case 16 + 0: f = 3.0f * zp[2] - 1.0f; df = 6.0f * zp[1]; break;
    case 16 + 1: f = zp[1]; df = 1.0f; break;
    case 16 + 2: f = 1.0f; df = 0.0f; break;
    case 24 + 0: f = 5.0f * zp[3] - 3.0f * zp[1]; df = 15.0f * zp[2] - 3.0f; break;
    case 24 + 1: f = 5.0f * zp[2] - 1.0f; df = 10.0f * zp[1]; break;
    case 24 + 2: f = zp[1]; df = 1.0f; break;
    case 24 + 3: f = 1.0f; df = 0.0f; break;
    case 32 + 0: f = 35.0f * zp[4] - 30.0f * zp[2] + 3.0f; df = 140.0f * zp[3] - 60.0f * zp[1]; break;
    case 32 + 1: f = 7.0f * zp[3] - 3.0f * zp[1]; df = 21.0f * zp[2] - 3.0f; break;
    case 32 + 2: f = 7.0f * zp[2] - 1.0f; df = 14.0f * zp[1]; break;
    case 32 + 3: f = zp[1]; df = 1.0f; break;
    case 32 + 4: f = 1.0f; df = 0.0f; break;
    default: break;
  }
  *dzf = df;
  return f;
}

}  // namespace nepx
