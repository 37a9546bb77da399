// nep_force.cu -- NEP energy, force and virial on sm_100a.
//
// Three kernels per force call (four where k_angular_f12 runs by itself), each
// giving a group of G lanes to one center (4 to 32: engine_choose).  Every phase is local to the group, so no CTA-wide barrier
// follows the set-up (except in the tensor-core ANN, whose MMAs span the
// CTA's centers).
//
//  k_filter_radial  one sweep over the center's sorted Verlet row applies the
//    reference's FP32 typewise predicate (nep.cu:503-561), writes the radial
//    and angular rows in order (group ballot + popcount) and sums the radial
//    descriptors q_n = sum_j sum_k c(ti,tj)[n][k] f_k(d_ij) through per-type
//    bins of the basis values.
//  k_nep_fused  (descriptors + ANN)
//    1. the radial descriptors (explicit rows: evaluated here);
//    2. a sweep over the dense angular row accumulates the moments
//       s[n][lm] = sum_j g_n(d_ij) Y_lm(r_ij/d) in registers; a register
//       reduce-scatter across the group lands each lane's share in shared
//       memory;
//    3. per center: invariants q_L and q_222/q_1111/q_112/q_123/q_233/q_134,
//       the one-hidden-layer ANN (site energy, dE/dq), the moment derivatives
//       a[n][lm] = dE/ds[n][lm], and the radial force coefficients
//       alpha[t][k] = sum_n dE/dq_n c(ti,t)[n][k] (stored for the gather).
//    Mixed precision runs the ANN of the CTA's centers as two tcgen05 MMAs
//    (16-bit operands, FP32 accumulators in TMEM, tc_ann) in place of the
//    per-center FP32 contraction.  Reference: find_descriptor (nep.cu:569-748).
//  k_angular_f12  each directed partial force
//       f12(i,j) = (sum_lm B_lm Y_lm) r^ + (1/d)(I - r^r^T) sum_lm A_lm dY_lm/dr^
//    with A_lm = sum_n a[n][lm] g_n and B_lm = sum_n a[n][lm] g'_n: the
//    harmonic ladder runs once per edge, not once per (edge, n) as in
//    accumulate_f12 (nep_utilities.cuh:1240-1491).  Reference:
//    find_partial_force_angular (nep.cu:890-991).
//  k_gather  radial pair force from both site energies with the per-atom
//    alpha coefficients (w_ij = sum_k f'_k(d) alpha_i[tj][k]), the angular
//    exchange F_i += f12(i,j) - f12(j,i) with the reverse slot found in j's
//    sorted row through its row of heads (reverse_slot; explicit rows: both
//    directed forces evaluated here), ZBL, and the per-atom virial W_i = sum_j r_ij (x) f_ji.
//    Reference: find_force_radial (nep.cu:756-881), gpu_find_force_many_body
//    (potential.cu:81-210), find_force_ZBL (nep.cu:996-1111).
//
// Harmonic degree: instances for l_max <= 4 (24 moment components per n) and
// l_max 5..8 (80 components).
#include <cstdio>
#include <mutex>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <utility>

#include "engine.h"
#include "harmonic_tables.h"
#include "invariants.h"
#include "tcgen05.cuh"

namespace nepx {

namespace {

constexpr int kBlock = 128;      // threads per CTA
constexpr int kChunkN = 5;       // radial functions per angular-moment sweep (3 CTAs per SM)
constexpr int kChunkN4 = 3;      // the same at 4 CTAs per SM (fewer live accumulators)
constexpr unsigned kFull = 0xffffffffu;

// Weights of the three-body invariants q_L and coefficients of the
// z-polynomials of the harmonics, degrees 1..8 (harmonic_tables.h; the
// reference's C3B and Z_COEFFICIENT_L tables, nep_utilities.cuh:51-187).
__constant__ float c_C3B[kNumLMHigh];
__constant__ float c_Zc[kHarmonicLMax + 1][kHarmonicLMax + 1][kHarmonicLMax + 1];

template <int LMAX>
__host__ __device__ constexpr int num_lm() { return (LMAX + 1) * (LMAX + 1) - 1; }

// Z_Lm(z) and dZ_Lm/dz with zp[k] = z^k; degrees above 4 from c_Zc.
__device__ __forceinline__ float zpoly_any(int L, int m, const float* zp, float* dzf)
{
  if (L <= 4) return zpoly(L, m, zp, dzf);
  float f = 0.0f, df = 0.0f;
#pragma unroll
  for (int k = 0; k <= kHarmonicLMax; ++k) {
    if (k <= L - m && ((L - m - k) & 1) == 0) {
      const float c = c_Zc[L][m][k];
      f += c * zp[k];
      if (k > 0) df += c * static_cast<float>(k) * zp[k - 1];
    }
  }
  *dzf = df;
  return f;
}

// Harmonics Y[lm], lm < (L_max + 1)^2 - 1, at the unit vector u, degrees up
// to LMAX (the instance's bound) and L_max (the model's), handed one at a
// time to f(lm, Y[lm]) with lm a compile-time index once unrolled (no array
// of all harmonics stays live).
template <int LMAX, typename F>
__device__ __forceinline__ void for_each_harmonic(int L_max, float ux, float uy, float uz, F&& f)
{
  float zp[LMAX + 1];
  zp[0] = 1.0f;
#pragma unroll
  for (int k = 1; k <= LMAX; ++k) zp[k] = zp[k - 1] * uz;
  int idx = 0;
#pragma unroll
  for (int L = 1; L <= LMAX; ++L) {
    if (L > L_max) break;
    float re = ux, im = uy;
#pragma unroll
    for (int m = 0; m <= L; ++m) {
      float dzf;
      const float zf = zpoly_any(L, m, zp, &dzf);
      if (m == 0) {
        f(idx++, zf);
      } else {
        f(idx++, zf * re);
        f(idx++, zf * im);
        const float r2 = ux * re - uy * im;
        im = ux * im + uy * re;
        re = r2;
      }
    }
  }
}

// Many-body invariants as monomials c * s[i0] s[i1] s[i2] (s[i3]) of the raw
// moments, transcribed from the polynomials of find_q
// (nep_utilities.cuh:1661-1728).  c_inv_start[v] .. c_inv_start[v+1] are the
// monomials of invariant v.
struct Monomial {
  float c;
  signed char i[4];
};
__constant__ Monomial c_mono[128];
__constant__ int c_inv_start[kMaxInv + 1];

// The same invariants for degrees <= 4 in registers: the monomial list of
// invariant ID (invariants.h) unrolled at compile time, so s and the
// derivatives a are register arrays of the 24 moment components of one n.
// Value: sum over monomials of c s[i0] s[i1] s[i2] (s[i3]), in list order.
template <int ID, int M>
__device__ __forceinline__ float inv_term(const float (&s)[kNumLM])
{
  constexpr InvMono mo = inv_mono(ID, M);
  float t = mo.c * s[mo.a] * s[mo.b] * s[mo.cc];
  if constexpr (mo.d >= 0) t *= s[mo.d];
  return t;
}

template <int ID, int... M>
__device__ __forceinline__ float inv_value(const float (&s)[kNumLM],
                                           std::integer_sequence<int, M...>)
{
  float acc = 0.0f;
  ((acc += inv_term<ID, M>(s)), ...);
  return acc;
}

template <int I>
__device__ __forceinline__ float inv_value_of(const float (&s)[kNumLM])
{
  return inv_value<I>(s, std::make_integer_sequence<int, inv_count(I)>{});
}

// Derivative terms: for every factor Q of monomial M, f c times the other
// factors in list order, added to a[factor Q].
template <int ID, int M, int Q, int R>
__device__ __forceinline__ float inv_grad_prod(const float (&s)[kNumLM], float t)
{
  constexpr InvMono mo = inv_mono(ID, M);
  constexpr int nf = mo.d >= 0 ? 4 : 3;
  if constexpr (R >= nf) {
    return t;
  } else {
    constexpr int i = R == 0 ? mo.a : R == 1 ? mo.b : R == 2 ? mo.cc : mo.d;
    if constexpr (R != Q) t *= s[i];
    return inv_grad_prod<ID, M, Q, R + 1>(s, t);
  }
}

template <int ID, int M, int Q>
__device__ __forceinline__ void inv_grad_factor(const float (&s)[kNumLM], float (&a)[kNumLM],
                                                float f)
{
  constexpr InvMono mo = inv_mono(ID, M);
  constexpr int nf = mo.d >= 0 ? 4 : 3;
  if constexpr (Q < nf) {
    constexpr int i = Q == 0 ? mo.a : Q == 1 ? mo.b : Q == 2 ? mo.cc : mo.d;
    a[i] += inv_grad_prod<ID, M, Q, 0>(s, f * mo.c);
    inv_grad_factor<ID, M, Q + 1>(s, a, f);
  }
}

template <int ID, int... M>
__device__ __forceinline__ void inv_grad(const float (&s)[kNumLM], float (&a)[kNumLM], float f,
                                         std::integer_sequence<int, M...>)
{
  (inv_grad_factor<ID, M, 0>(s, a, f), ...);
}

template <int I>
__device__ __forceinline__ void inv_grad_of(const float (&s)[kNumLM], float (&a)[kNumLM], float f)
{
  inv_grad<I>(s, a, f, std::make_integer_sequence<int, inv_count(I)>{});
}

// runtime invariant id -> its unrolled form
__device__ __forceinline__ float inv_value_id(int id, const float (&s)[kNumLM])
{
  switch (id) {
    case 0: return inv_value_of<0>(s);
    case 1: return inv_value_of<1>(s);
    case 2: return inv_value_of<2>(s);
    case 3: return inv_value_of<3>(s);
    case 4: return inv_value_of<4>(s);
    default: return inv_value_of<5>(s);
  }
}

__device__ __forceinline__ void inv_grad_id(int id, const float (&s)[kNumLM], float (&a)[kNumLM],
                                            float f)
{
  switch (id) {
    case 0: inv_grad_of<0>(s, a, f); break;
    case 1: inv_grad_of<1>(s, a, f); break;
    case 2: inv_grad_of<2>(s, a, f); break;
    case 3: inv_grad_of<3>(s, a, f); break;
    case 4: inv_grad_of<4>(s, a, f); break;
    default: inv_grad_of<5>(s, a, f); break;
  }
}

// The 24 moments of one n from shared memory (16-byte aligned) and back.
__device__ __forceinline__ void load24(const float* src, float (&v)[kNumLM])
{
#pragma unroll
  for (int q = 0; q < kNumLM / 4; ++q) {
    const float4 x = reinterpret_cast<const float4*>(src)[q];
    v[4 * q] = x.x;
    v[4 * q + 1] = x.y;
    v[4 * q + 2] = x.z;
    v[4 * q + 3] = x.w;
  }
}

__device__ __forceinline__ void store24(float* dst, const float (&v)[kNumLM])
{
#pragma unroll
  for (int q = 0; q < kNumLM / 4; ++q)
    reinterpret_cast<float4*>(dst)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2],
                                                    v[4 * q + 3]);
}

#include "zbl.cuh"

__host__ __device__ constexpr int round4(int x) { return (x + 3) & ~3; }

// Shared-memory layout of k_nep_fused (in floats; the tensor-core region in bytes).
struct FusedLayout {
  int kpr, kpa;        // basis sizes padded to float4
  int c_rad, c_ang;    // coefficient tables [T*T][n][kp]
  int cut_r, cut_a;    // pair cutoffs and reciprocals [T*T] float2, radial and angular
  int wt;              // transposed ANN weights [T][dim][H4], or -1: read from global
  int per_atom;        // floats of per-center scratch
  int s, a, q, fp, gh; // offsets inside one center's scratch
  int atoms_base;      // offset of the per-center scratch
  int total_bytes;
  // tensor-core ANN (byte offsets from the start): 16-bit tiles of one chunk
  // of 128 stacked hidden units, W0 [128][dimk] and W0^T [dim][128], the CTA's
  // descriptors [APB][dimk] and hidden-layer derivatives [APB][128]; energy
  // partials [4][APB]; per type, the bit mask of the CTA's centers of that
  // type [kMaxTypes]; the mbarrier, the TMEM address and a flag
  int tc_w, tc_wt, tc_q, tc_g, tc_e, tc_type, tc_bar, tc_misc;
};

// Shared memory one CTA may use with the ANN weights staged, when `minb`
// CTAs share an SM (228 KB per SM, 1 KB of it reserved per CTA).
__host__ __device__ constexpr int fused_smem_budget(int minb) { return 228 * 1024 / minb - 1024; }

// kp: row stride of the coefficient tables, the padded basis size of the
// kernel instance (rows are zero-filled up to it, so float4 dot products of
// the full compile-time width stay inside the row).
// tc: the layout of the tensor-core ANN build (16-bit tiles first, no FP32
// weights staged, no per-center hidden-unit scratch).  An MMA reads 128 rows
// of its A tile: rows past the stacked hidden units (or dim) are read from
// whatever follows in shared memory and only feed accumulator rows the
// epilogue never reads, so total_bytes covers the 128-row span of both A tiles.
__host__ __device__ inline FusedLayout fused_layout(const ModelParams& p, int atoms_per_block,
                                                   int kp, int budget, bool tc = false)
{
  FusedLayout L;
  L.kpr = kp;
  L.kpa = kp;
  const int tt = p.T * p.T;
  int base = 0;   // floats before the tables
  if (tc) {
    auto up128 = [](int x) { return (x + 127) & ~127; };
    const int dimk = p.tc_dimk, th = p.T * p.H;
    const int rows = ((th < 128 ? th : 128) + 7) & ~7;
    L.tc_w = 0;
    L.tc_wt = up128(L.tc_w + rows * dimk * 2);
    L.tc_q = up128(L.tc_wt + ((p.dim + 7) & ~7) * 128 * 2);
    L.tc_g = up128(L.tc_q + atoms_per_block * dimk * 2);
    L.tc_e = up128(L.tc_g + atoms_per_block * 128 * 2);
    L.tc_type = L.tc_e + 4 * atoms_per_block * 4;
    L.tc_bar = (L.tc_type + kMaxTypes * 4 + 7) & ~7;
    L.tc_misc = L.tc_bar + 8;
    base = up128(L.tc_misc + 16) / 4;
  } else {
    L.tc_w = L.tc_wt = L.tc_q = L.tc_g = L.tc_e = L.tc_type = L.tc_bar = L.tc_misc = -1;
  }
  L.c_rad = base;
  L.c_ang = L.c_rad + tt * p.nR * L.kpr;
  L.s = 0;
  L.a = p.nA * p.nlm;
  L.q = 2 * p.nA * p.nlm;
  L.fp = L.q + round4(p.dim);
  L.gh = L.fp + round4(p.dim);
  // per-center stride: 16-byte aligned (float4 reads of the a[n][lm] rows)
  // and an odd number of 16-byte units, so float4 rows of neighbouring
  // centers start on different banks
  L.per_atom = round4(L.gh + (tc ? 0 : p.H));
  if ((L.per_atom / 4) % 2 == 0) L.per_atom += 4;
  L.cut_r = round4(L.c_ang + tt * p.nA * L.kpa);
  L.cut_a = L.cut_r + 2 * tt;
  const int tables = round4(L.cut_a + 2 * tt);
  const int wsize = p.T * p.dim * p.H4;
  L.wt = tables;
  L.atoms_base = tables + wsize;
  L.total_bytes = 4 * (L.atoms_base + atoms_per_block * L.per_atom);
  if (tc || L.total_bytes > budget) {   // weights stay in global memory
    L.wt = -1;
    L.atoms_base = tables;
    L.total_bytes = 4 * (L.atoms_base + atoms_per_block * L.per_atom);
  }
  if (tc) {
    const int need_w = L.tc_w + 128 * p.tc_dimk * 2, need_wt = L.tc_wt + 128 * 128 * 2;
    L.total_bytes = (L.total_bytes > need_w ? L.total_bytes : need_w);
    L.total_bytes = (L.total_bytes > need_wt ? L.total_bytes : need_wt);
    L.total_bytes = (L.total_bytes + 15) & ~15;
  }
  return L;
}

// Cutoffs of the type pairs and their correctly rounded reciprocals (computed on
// the host, ModelParams::pair_cut) in shared memory, [T*T] of (cutoff, 1 /
// cutoff): which 0 radial, 1 angular.  An edge reads its pair in one access.
__device__ __forceinline__ void load_pair_cut(const ModelParams& p, int which, float2* dst)
{
  const int tt = p.T * p.T;
  for (int k = threadIdx.x; k < tt; k += blockDim.x)
    dst[k] = make_float2(__ldg(p.pair_cut + 2 * which * tt + k),
                         __ldg(p.pair_cut + (2 * which + 1) * tt + k));
}

// f[k] . c[k] over KM basis values with float4 loads of a padded row, in
// packed pairs for the short basis (the long one's pairs cost more register
// moves than they save: 13,824 carbon atoms at basis 16/12, descriptor stage
// 238 us scalar, 249 us packed).
template <int KM>
__device__ __forceinline__ float dot_basis(const float* __restrict__ c, const float* f)
{
  if constexpr (KM > 9) {
    float acc = 0.0f;
#pragma unroll
    for (int q = 0; q < (KM + 3) / 4; ++q) {
      const float4 cv = *reinterpret_cast<const float4*>(c + 4 * q);
      acc += cv.x * f[4 * q] + cv.y * f[4 * q + 1] + cv.z * f[4 * q + 2] + cv.w * f[4 * q + 3];
    }
    return acc;
  }
  float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int q = 0; q < (KM + 3) / 4; ++q) {
    const float4 cv = *reinterpret_cast<const float4*>(c + 4 * q);
    const float2 lo = make_float2(cv.x, cv.y), f01 = make_float2(f[4 * q], f[4 * q + 1]);
    acc = q == 0 ? mul2(lo, f01) : fma2(lo, f01, acc);
    // the last row part past the basis is zero
    if (4 * q + 2 < KM) acc = fma2(make_float2(cv.z, cv.w), make_float2(f[4 * q + 2], f[4 * q + 3]), acc);
  }
  return acc.x + acc.y;
}

// Shared memory of k_filter_radial: the coefficient table, then per-lane
// type bins of the basis sums when T * kp <= kFilterBinMax floats.
constexpr int kFilterBinMax = 48;
__host__ __device__ inline int filter_table_floats(const ModelParams& p, int kp)
{
  return round4(p.T * p.T * p.nR * kp);
}
__host__ __device__ inline int filter_bin_float4(const ModelParams& p, int kp)
{
  const int q = p.T * kp / 4;
  return q | 1;
}
// Where the filter keeps its bins (BIN): nowhere (the contraction per edge),
// shared memory, or registers: one type and the short basis (10 of them; two
// types' 20, or the long basis's 18, cost more than they save: water 24k
// descriptor stage 114 us with shared bins, 123 us with registers).
constexpr int kBinNone = 0, kBinShared = 1, kBinRegs = 2;
template <int KM>
int filter_bin(const ModelParams& p)
{
  if (p.T == 1 && KM <= 9) return kBinRegs;
  return p.T * ((KM + 3) & ~3) <= kFilterBinMax ? kBinShared : kBinNone;
}

// Neighbour type of an edge record (float4: displacement, type << 28 | index).
__device__ __forceinline__ int row_type(const float4& e)
{
  return static_cast<int>(static_cast<unsigned>(__float_as_int(e.w)) >> kRowTypeShift);
}

// group ballot: the bits of the G lanes of this lane's group
template <int G>
__device__ __forceinline__ unsigned group_ballot(bool pred, int group)
{
  const unsigned b = __ballot_sync(kFull, pred);
  if constexpr (G == 32) return b;
  else return (b >> (group * G)) & ((1u << G) - 1u);
}

template <int G>
__device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Reduce-scatter of L values across the G lanes of a group: afterwards lane
// gl holds the group sums of v[base .. base + L/G) in v[0 .. L/G).
template <int L, int O>
__device__ __forceinline__ void rs_step(float* v, int gl, int& base)
{
  constexpr int half = L / 2;
  const bool hi = (gl & O) != 0;
#pragma unroll
  for (int i = 0; i < half; ++i) {
    const float send = hi ? v[i] : v[i + half];
    const float keep = hi ? v[i + half] : v[i];
    v[i] = keep + __shfl_xor_sync(kFull, send, O);
  }
  if (hi) base += half;
}

template <int G, int L>
__device__ __forceinline__ int reduce_scatter(float* v, int gl)
{
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "group of 4 to 32 lanes");
  static_assert(L % G == 0, "share must divide evenly");
  int base = 0;
  if constexpr (G == 32) {
    rs_step<L, 16>(v, gl, base);
    rs_step<L / 2, 8>(v, gl, base);
    rs_step<L / 4, 4>(v, gl, base);
    rs_step<L / 8, 2>(v, gl, base);
    rs_step<L / 16, 1>(v, gl, base);
  } else if constexpr (G == 16) {
    rs_step<L, 8>(v, gl, base);
    rs_step<L / 2, 4>(v, gl, base);
    rs_step<L / 4, 2>(v, gl, base);
    rs_step<L / 8, 1>(v, gl, base);
  } else if constexpr (G == 8) {
    rs_step<L, 4>(v, gl, base);
    rs_step<L / 2, 2>(v, gl, base);
    rs_step<L / 4, 1>(v, gl, base);
  } else {
    rs_step<L, 2>(v, gl, base);
    rs_step<L / 2, 1>(v, gl, base);
  }
  return base;
}

// Row stride of alpha: the padded basis, or for the long basis whole 32-byte
// sectors, so that a neighbour's row is read with 32-byte loads (gather of 13,824
// carbon atoms at basis 16: 74 -> 70 us; for the short basis's nine values they
// cost: 1M carbon 1.19 -> 1.23 ms).
template <int KM>
__host__ __device__ constexpr int alpha_row() { return KM <= 9 ? round4(KM) : (KM + 7) & ~7; }

// sum_k f[k] alpha[k] over KM basis values of a row of alpha in global memory.
template <int KM>
__device__ __forceinline__ float dot_alpha(const float* __restrict__ al, const float* f)
{
  if constexpr (KM <= 9) return dot_basis<KM>(al, f);
  float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int q = 0; q + 8 <= KM; q += 8) {
    float a[8];
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]),
          "=f"(a[7])
        : "l"(al + q));
#pragma unroll
    for (int r = 0; r < 8; r += 2)
      acc = fma2(make_float2(a[r], a[r + 1]), make_float2(f[q + r], f[q + r + 1]), acc);
  }
  float sum = acc.x + acc.y;
#pragma unroll
  for (int k = KM & ~7; k < KM; ++k) sum = fmaf(__ldg(al + k), f[k], sum);
  return sum;
}

// Radial force coefficients of one center, alpha[t][k] = sum_n Fp[n] c(t1,t)[n][k]
// (the group's lanes split the T * kpr entries; rows of `row` floats); c_rad:
// shared-memory table.
template <int G>
__device__ __forceinline__ void center_alpha(int T, int nR, int t1, const float* s_fp,
                                             const float* c_rad, int kpr, int row, int gl,
                                             float* al)
{
  for (int e = gl; e < T * kpr; e += G) {
    const int t = e / kpr, kk = e % kpr;
    const float* c = c_rad + (t1 * T + t) * nR * kpr + kk;
    float acc = 0.0f;
    for (int n = 0; n < nR; ++n) acc += s_fp[n] * c[n * kpr];
    al[t * row + kk] = acc;
  }
}

// Moment derivatives of one center, a[n][lm] = dE/ds[n][lm] (one lane owns
// one n); the monomial terms read the moments at run-time indices, so both
// live in shared memory.
template <int G, int NLM>
__device__ __forceinline__ void center_acoef(const ModelParams& p, int nR, int nA, int L_max,
                                             const float* s_s, float* s_a, const float* s_fp,
                                             int gl)
{
  if constexpr (NLM == kNumLM) {
    // degrees <= 4: moments and derivatives of one n in registers
    const float* fp = s_fp + nR;
    for (int n = gl; n < nA; n += G) {
      float sv[kNumLM], av[kNumLM];
      load24(s_s + n * NLM, sv);
#pragma unroll
      for (int Lq = 1; Lq <= 4; ++Lq) {
        const int st0 = Lq * Lq - 1;
        const bool on = Lq <= L_max;
        const float f = on ? fp[(Lq - 1) * nA + n] : 0.0f;
        av[st0] = on ? 2.0f * f * c_C3B[st0] * sv[st0] : 0.0f;
#pragma unroll
        for (int k = 1; k < 2 * Lq + 1; ++k)
          av[st0 + k] = on ? 4.0f * f * c_C3B[st0 + k] * sv[st0 + k] : 0.0f;
      }
      int col = L_max;
      for (int w = 0; w < p.num_inv; ++w, ++col)
        inv_grad_id(p.inv_id[w], sv, av, fp[col * nA + n]);
      store24(s_a + n * NLM, av);
    }
  } else {
    for (int n = gl; n < nA; n += G) {
      const float* sv = s_s + n * NLM;
      float* av = s_a + n * NLM;
      const float* fp = s_fp + nR;
      int col = 0;
      for (int Lq = 1; Lq <= L_max; ++Lq, ++col) {
        const int st0 = Lq * Lq - 1;
        const float f = fp[col * nA + n];
        av[st0] = 2.0f * f * c_C3B[st0] * sv[st0];
        for (int k = 1; k < 2 * Lq + 1; ++k) av[st0 + k] = 4.0f * f * c_C3B[st0 + k] * sv[st0 + k];
      }
      for (int lm = (L_max + 1) * (L_max + 1) - 1; lm < NLM; ++lm) av[lm] = 0.0f;
      for (int w = 0; w < p.num_inv; ++w, ++col) {
        const int id = p.inv_id[w];
        const float f = fp[col * nA + n];
        for (int m = c_inv_start[id]; m < c_inv_start[id + 1]; ++m) {
          const Monomial mo = c_mono[m];
          const int nf = mo.i[3] >= 0 ? 4 : 3;
          for (int a = 0; a < nf; ++a) {
            float t = f * mo.c;
            for (int r = 0; r < nf; ++r)
              if (r != a) t *= sv[mo.i[r]];
            av[mo.i[a]] += t;
          }
        }
      }
    }
  }
}

// tanh of the mixed-precision ANN: the hardware approximation (PTX
// tanh.approx.f32, relative error about 2^-11, the size of an FP16 operand's
// rounding).
__device__ __forceinline__ float tanh_fast(float x)
{
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One FP32 value as a 16-bit MMA operand (FP16 or BF16, round to nearest).
__device__ __forceinline__ void store16(unsigned char* at, float v, bool bf16)
{
  *reinterpret_cast<unsigned short*>(at) =
    bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

// One chunk of the stacked weights into the tiles (16-byte rows of core
// matrices): rows m = 128 k .. of W0 (stacked m = t H + h) and columns
// 128 k .. of W0^T.
__device__ __forceinline__ void tc_stage_chunk(const ModelParams& p, const FusedLayout& Lay,
                                               unsigned char* smb, int k)
{
  const int dimk = p.tc_dimk, th = p.T * p.H, m0 = 128 * k;
  const int rows = th - m0 < 128 ? th - m0 : 128;
  const int cw = dimk / 8;
  const uint4* w = reinterpret_cast<const uint4*>(p.w0h + static_cast<size_t>(m0) * dimk);
  for (int e = threadIdx.x; e < rows * cw; e += kBlock)
    *reinterpret_cast<uint4*>(smb + Lay.tc_w + tc::off16(e / cw, 8 * (e % cw), dimk)) =
      __ldg(w + e);
  for (int e = threadIdx.x; e < p.dim * 16; e += kBlock) {
    const int d = e / 16, c = e % 16;
    *reinterpret_cast<uint4*>(smb + Lay.tc_wt + tc::off16(d, 8 * c, 128)) =
      __ldg(reinterpret_cast<const uint4*>(p.w0th + static_cast<size_t>(d) * p.tc_kt + m0 +
                                           8 * c));
  }
}

// Tensor-core set-up of a CTA of the mixed-precision descriptor kernel (before
// its first barrier): TMEM for the two accumulators, the mbarrier, flags, and
// with a single chunk of stacked hidden units the weight tiles.
template <int APB>
__device__ __forceinline__ void tc_ann_setup(const ModelParams& p, const FusedLayout& Lay,
                                             unsigned char* smb)
{
  constexpr int kCols = 2 * APB < 32 ? 32 : 2 * APB;   // D1 | D2, APB columns each
  uint32_t* misc = reinterpret_cast<uint32_t*>(smb + Lay.tc_misc);
  if (threadIdx.x < 32) tc::tmem_alloc(misc + 2, kCols);
  if (threadIdx.x == 0) {
    tc::mbar_init(tc::smem_u32(smb + Lay.tc_bar));
    misc[0] = 0u;   // largest |q| of the CTA (float bits)
  }
  unsigned* tmask = reinterpret_cast<unsigned*>(smb + Lay.tc_type);
  if (threadIdx.x < kMaxTypes) tmask[threadIdx.x] = 0u;   // centers of each type
  if (p.tc_kt == 128) {
    tc_stage_chunk(p, Lay, smb, 0);
    tc::fence_async_smem();
  }
}

// The per-atom ANN of all APB centers of the CTA on the tensor cores (whole
// CTA; s_q of every center holds its scaled descriptors).  The hidden units
// of all types are stacked, m = t H + h, and run in chunks of 128:
//   GEMM1 (M = 128 stacked units, N = APB centers, K = dim):
//     Z = W0 Q^T, from the 16-bit tiles of W0 * sw and Q * sq;
//   epilogue (thread = unit m = its TMEM lane, t = m / H): for the centers of
//     type t, x = tanh(z / (sw sq) - b0) (hardware tanh), E += w1 x,
//     G = w1 (1 - x^2) * sg (zero for the other centers);
//   GEMM2 (M = dim, N = APB, K = the chunk's 128 units): dE/dq += W0^T G^T,
//     accumulated over the chunks in TMEM.
// sw, sg are the model's power-of-two scales (nepx_set_precision), sq the
// CTA's (largest |q| to 2^14): in FP16 every operand keeps its 11-bit
// significand; unscaling by powers of two is exact.  Then each center's
// dE/dq (times q_scaler) lands in its s_fp and its site energy in pe_ann.
// Every wait is bounded: a timeout sets ann_error, waits (bounded again) for
// the MMAs in flight and lets the CTA finish with the error flagged.
template <int APB, int G>
__device__ void tc_ann(const ModelParams& p, const FusedLayout& Lay, float* sm, int slot,
                       int gl, bool active, int t1, int i, const float* s_q,
                       double* __restrict__ pe_ann, NeighborState* st)
{
  constexpr int kCols = 2 * APB < 32 ? 32 : 2 * APB;
  unsigned char* smb = reinterpret_cast<unsigned char*>(sm);
  unsigned char* Wt = smb + Lay.tc_w;
  unsigned char* Vt = smb + Lay.tc_wt;
  unsigned char* Qt = smb + Lay.tc_q;
  unsigned char* Gt = smb + Lay.tc_g;
  float* s_e = reinterpret_cast<float*>(smb + Lay.tc_e);
  unsigned* s_tmask = reinterpret_cast<unsigned*>(smb + Lay.tc_type);
  uint32_t* misc = reinterpret_cast<uint32_t*>(smb + Lay.tc_misc);
  const uint32_t bar = tc::smem_u32(smb + Lay.tc_bar);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int H = p.H, dim = p.dim, dimk = p.tc_dimk, th = p.T * H;
  const int chunks = p.tc_kt / 128;
  const bool bf16 = p.tc_bf16 != 0;

  // the CTA's largest |q| and the center types
  float qm = 0.0f;
  if (active)
    for (int d = gl; d < dim; d += G) qm = fmaxf(qm, fabsf(s_q[d]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) qm = fmaxf(qm, __shfl_xor_sync(kFull, qm, o));
  if (lane == 0) atomicMax(reinterpret_cast<int*>(misc), __float_as_int(qm));
  if (gl == 0 && active) atomicOr(s_tmask + t1, 1u << slot);
  __syncthreads();
  const float qmax = __int_as_float(static_cast<int>(misc[0]));
  int ex = 0;
  frexpf(qmax, &ex);
  const float sq = qmax > 0.0f ? ldexpf(1.0f, max(-60, min(60, 14 - ex))) : 1.0f;
  // this center's row of the descriptor tile, zero past dim and for idle slots
  for (int d = gl; d < dimk; d += G)
    store16(Qt + tc::off16(slot, d, dimk), (active && d < dim) ? s_q[d] * sq : 0.0f, bf16);
  tc::fence_async_smem();
  const uint32_t tmem = misc[2];
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  const uint32_t id = tc::idesc_f16(128, APB, bf16);
  const float unscale1 = 1.0f / (sq * p.tc_sw), unscale2 = 1.0f / (p.tc_sw * p.tc_sg);
  float e_acc[APB];
#pragma unroll
  for (int c = 0; c < APB; ++c) e_acc[c] = 0.0f;
  uint32_t phase = 0;
  bool failed = false;
  for (int k = 0; k < chunks; ++k) {
    if (chunks > 1) {
      // the previous chunk's MMAs are complete: its tiles may be overwritten
      tc_stage_chunk(p, Lay, smb, k);
      tc::fence_async_smem();
    }
    tc::before_sync();
    __syncthreads();
    tc::after_sync();
    if (tid == 0) {
      for (int s = 0; s < dimk / 16; ++s) {
        const uint64_t a = tc::smem_desc(tc::smem_u32(Wt + tc::off16(0, 16 * s, dimk)), dimk);
        const uint64_t b = tc::smem_desc(tc::smem_u32(Qt + tc::off16(0, 16 * s, dimk)), dimk);
        tc::mma_f16(tmem, a, b, id, s > 0 ? 1u : 0u);
      }
      tc::mma_commit(bar);
    }
    bool ok = tc::mbar_wait(bar, phase);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    tc::after_sync();
    const int m = 128 * k + tid;
    const bool unit = m < th;
    const unsigned mine = unit ? s_tmask[m / H] : 0u;   // the centers of this unit's type
    const float b0m = unit ? __ldg(p.b0 + m) : 0.0f;   // b0 and w1 are [T][H]: index m
    const float w1m = unit ? __ldg(p.w1 + m) : 0.0f;
#pragma unroll
    for (int c0 = 0; c0 < APB; c0 += 16) {
      float z[16];
      tc::tmem_ld16(lane_addr + c0, z);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int c = c0 + q;
        float g = 0.0f;
        if ((mine >> c) & 1u) {
          const float x = tanh_fast(z[q] * unscale1 - b0m);
          e_acc[c] += w1m * x;
          g = w1m * (1.0f - x * x) * p.tc_sg;
        }
        store16(Gt + tc::off16(c, tid, 128), g, bf16);
      }
    }
    tc::fence_async_smem();
    tc::before_sync();
    __syncthreads();   // G complete, D1 read
    tc::after_sync();
    if (tid == 0) {
      for (int s = 0; s < 128 / 16; ++s) {
        const uint64_t a = tc::smem_desc(tc::smem_u32(Vt + tc::off16(0, 16 * s, 128)), 128);
        const uint64_t b = tc::smem_desc(tc::smem_u32(Gt + tc::off16(0, 16 * s, 128)), 128);
        tc::mma_f16(tmem + APB, a, b, id, (k > 0 || s > 0) ? 1u : 0u);
      }
      tc::mma_commit(bar);
    }
    ok = tc::mbar_wait(bar, phase);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    tc::after_sync();
  }
  if (!failed) {
    // dE/dq: descriptor component d = this thread's TMEM lane, every center
    const int d = tid;
    const float qs = d < dim ? __ldg(p.q_scaler + d) : 0.0f;
#pragma unroll
    for (int c0 = 0; c0 < APB; c0 += 16) {
      float f[16];
      tc::tmem_ld16(lane_addr + APB + c0, f);
      if (d < dim)
#pragma unroll
        for (int q = 0; q < 16; ++q)
          sm[Lay.atoms_base + (c0 + q) * Lay.per_atom + Lay.fp + d] = f[q] * unscale2 * qs;
    }
  }
  // site energies: each warp's partial sums over its 32 hidden units, lane c
  // ends with center c's (fixed order), then the four warps in order
  if constexpr (APB == 16) {
#pragma unroll
    for (int c = 0; c < 16; ++c) e_acc[c] += __shfl_xor_sync(kFull, e_acc[c], 16);
  }
  int at = 0;
  if constexpr (APB == 32) rs_step<32, 16>(e_acc, lane, at);
  rs_step<16, 8>(e_acc, lane, at);
  rs_step<8, 4>(e_acc, lane, at);
  rs_step<4, 2>(e_acc, lane, at);
  rs_step<2, 1>(e_acc, lane, at);
  if (lane < APB) s_e[warp * APB + at] = e_acc[0];
  if (failed) {
    if (tid == 0) atomicOr(&st->ann_error, 1);
    tc::mbar_wait(bar, phase ^ 1u);   // the MMAs of the phase that timed out
  }
  tc::before_sync();
  __syncthreads();
  tc::after_sync();
  if (warp == 0) tc::tmem_dealloc(misc[2], kCols);
  if (active && gl == 0) {
    const float e = s_e[slot] + s_e[APB + slot] + s_e[2 * APB + slot] + s_e[3 * APB + slot];
    pe_ann[i] = static_cast<double>(e - __ldg(p.out_bias + t1));
  }
}

// Typewise filter and radial descriptors (large-box path): one group of G
// lanes per center sweeps its sorted Verlet row with the next candidate's
// site in flight, applies the reference's FP32 predicate bit for bit (double
// difference rounded to float, float minimum image, the same x*x + y*y + z*z
// expression; nep.cu:503-561) and writes the radial and angular rows in
// order (group ballot + popcount), summing
// q_n = sum_j sum_k c(ti,tj)[n][k] f_k(d_ij) on the way.  BIN: each lane
// sums its edges' basis values per neighbour type, B[tj][k] += f_k(d_ij), and
// contracts them with c once at the end (q_n = sum_t sum_k c(ti,t)[n][k]
// B[t][k]) instead of the nR x kR contraction per edge.  The bins of one
// type are registers, those of several the lane's own shared memory (1M
// carbon, descriptor stage: 3.51 ms with shared bins, 3.48 with registers).
// Kept apart from k_nep_fused so this
// latency-bound sweep runs at the occupancy of its own register count.
// The length of an angular row and its every eighth entry also go to its row of
// heads, by which the gather finds an entry in two loads (reverse_slot).
// The angular edges are also written out, displacement and neighbour type, to
// the slots their forces f12 will take: the descriptor kernel then sweeps 16
// contiguous bytes per edge instead of fetching sites, and overwrites each
// slot with the force once it has read it.
// FAST: the mixed-precision build (hardware sqrt / reciprocal / sine-cosine
// approximations, see cutoff_fc), held to seven CTAs per SM (72 registers,
// as the exact build takes; it would take 78, rounded to 80: six CTAs).
template <int G, int NRM, int KM, int BIN, bool FAST>
__global__ void __launch_bounds__(kBlock, (FAST ? 7 : 0))
k_filter_radial(const ModelParams p, int N, const Box* __restrict__ box,
                const Site* __restrict__ sites, NeighborState* st,
                const int* __restrict__ nn_v, const int* __restrict__ nl_v, int mn_v,
                int* __restrict__ nn_r, int* __restrict__ nl_r, int mn_r,
                int* __restrict__ nn_a, int* __restrict__ nl_a, int mn_a,
                int st_a, int* __restrict__ heads, int st_h, float4* __restrict__ edges,
                float* __restrict__ qrad)
{
  constexpr int APW = 32 / G, APB = kBlock / G;
  constexpr int KP = (KM + 3) & ~3;
  extern __shared__ float sm[];   // radial coefficient table [T*T][nR][KP], then the bins
  const int tid = threadIdx.x;
  const int T = p.T, nR = p.nR, kR = p.kR;
  for (int k = tid; k < T * T * nR * KP; k += kBlock) {
    const int kk = k % KP, row = k / KP;
    sm[k] = kk < kR ? __ldg(p.c_pair + row * kR + kk) : 0.0f;
  }
  // this lane's bins [T][KP] (an odd number of float4 per lane: no bank conflicts)
  float4* bin = reinterpret_cast<float4*>(sm + filter_table_floats(p, KP)) +
                tid * filter_bin_float4(p, KP);
  if constexpr (BIN == kBinShared)
    for (int q = 0; q < T * KP / 4; ++q) bin[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (blockIdx.x == 0 && tid == 0) st->rebuild = 0;   // the Verlet list is consumed
  // per type pair: radial cutoff, its reciprocal, both cutoffs squared; then the
  // box's matrix
  float4* s_cut = reinterpret_cast<float4*>(
    sm + filter_table_floats(p, KP) +
    (BIN == kBinShared ? 4 * kBlock * filter_bin_float4(p, KP) : 0));
  for (int k = tid; k < T * T; k += kBlock) {
    const float rr = __ldg(p.pair_cut + k), ra = __ldg(p.pair_cut + 2 * T * T + k);
    s_cut[k] = make_float4(rr, __ldg(p.pair_cut + T * T + k), rr * rr, ra * ra);
  }
  const MinImage mic(box, reinterpret_cast<float*>(s_cut + T * T));
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5;
  const int group = lane / G, gl = lane % G;
  const int i = blockIdx.x * APB + warp * APW + group;
  const bool active = i < N;
  const Site me = active ? sites[i] : Site{0.0, 0.0, 0.0, 0};
  const double xi = me.x, yi = me.y, zi = me.z;
  const int t1 = BIN == kBinRegs ? 0 : static_cast<int>(me.type);
  const unsigned below = (1u << gl) - 1u;
  float qr[NRM];
#pragma unroll
  for (int n = 0; n < NRM; ++n) qr[n] = 0.0f;
  float rb[KP];
#pragma unroll
  for (int k = 0; k < KP; ++k) rb[k] = 0.0f;
  const int nv = active ? nn_v[i] : 0;
  const int nv_max = __reduce_max_sync(kFull, nv);
  const int* vrow = nl_v + static_cast<size_t>(i) * mn_v;
  int* rrow = nl_r + static_cast<size_t>(i) * mn_r;
  int* arow = nl_a + static_cast<size_t>(i) * st_a;
  int* hrow = heads + static_cast<size_t>(i) * st_h;
  float4* eout = edges + static_cast<size_t>(i) * mn_a;
  int cr = 0, ca = 0;
  // the next candidate's site and the index of the one after it in flight:
  // no load inside the loop waits on another
  int j_next = 0, j_after = 0;
  double2 sa_next = make_double2(0.0, 0.0), sc_next = make_double2(0.0, 0.0);
  if (gl < nv) {
    j_next = vrow[gl];
    site_load(sites, j_next, sa_next, sc_next);
  }
  if (gl + G < nv) j_after = vrow[gl + G];
  for (int base = 0; base < nv_max; base += G) {
    const int k = base + gl;
    const int j = j_next;
    const double2 sa = sa_next, sc = sc_next;
    if (k + G < nv) {
      j_next = j_after;
      site_load(sites, j_next, sa_next, sc_next);
    }
    if (k + 2 * G < nv) j_after = vrow[k + 2 * G];
    bool in_r = false, in_a = false;
    int t2 = 0;
    float x12 = 0.0f, y12 = 0.0f, z12 = 0.0f, d12_square = 0.0f, rc_radial = 1.0f;
    float rcinv_r = 1.0f;
    if (k < nv) {
      site_delta(mic, sa, sc, xi, yi, zi, x12, y12, z12, t2);
      if constexpr (BIN == kBinRegs) t2 = 0;   // one type: its cutoffs stay in registers
      d12_square = x12 * x12 + y12 * y12 + z12 * z12;
      const float4 cut = s_cut[t1 * T + t2];
      rc_radial = cut.x;
      rcinv_r = cut.y;
      in_r = d12_square < cut.z;
      in_a = in_r && d12_square < cut.w;
    }
    const unsigned mr = group_ballot<G>(in_r, group);
    const unsigned ma = group_ballot<G>(in_a, group);
    if (in_r) {
      const int at = cr + __popc(mr & below);
      if (at < mn_r) rrow[at] = j;
      float d, dinv;
      edge_length<FAST>(d12_square, d, dinv);
      const float rcinv = rcinv_r;
      float fc, fcp;
      cutoff_fc<FAST>(rc_radial, rcinv, d, fc, fcp);
      float fn[KP];
#pragma unroll
      for (int kk = 0; kk < KP; ++kk) fn[kk] = 0.0f;
      radial_basis<KM>(kR, rcinv, d, fc, fn);
      if constexpr (BIN == kBinRegs) {
#pragma unroll
        for (int k = 0; k < KM; ++k) rb[k] += fn[k];
      } else if constexpr (BIN == kBinShared) {
        float4* bt = bin + t2 * (KP / 4);
#pragma unroll
        for (int q = 0; q < KP / 4; ++q) {
          float4 v = bt[q];
          v.x += fn[4 * q];
          v.y += fn[4 * q + 1];
          v.z += fn[4 * q + 2];
          v.w += fn[4 * q + 3];
          bt[q] = v;
        }
      } else {
        const float* c = sm + (t1 * T + t2) * nR * KP;
#pragma unroll
        for (int n = 0; n < NRM; ++n)
          if (n < nR) qr[n] += dot_basis<KM>(c + n * KP, fn);
      }
    }
    if (in_a) {
      const int at = ca + __popc(ma & below);
      if (at < mn_a) {
        arow[at] = j;
        if (at % 8 == 0 && heads) hrow[1 + at / 8] = j;
        eout[at] = make_float4(x12, y12, z12, __int_as_float(t2 << kRowTypeShift));
      }
    }
    cr += __popc(mr);
    ca += __popc(ma);
  }
  if constexpr (BIN == kBinRegs) {
#pragma unroll
    for (int n = 0; n < NRM; ++n)
      if (n < nR) qr[n] += dot_basis<KM>(sm + n * KP, rb);
  } else if constexpr (BIN == kBinShared) {
    const float* bf = reinterpret_cast<const float*>(bin);
    for (int t = 0; t < T; ++t) {
      const float* c = sm + (t1 * T + t) * nR * KP;
#pragma unroll
      for (int n = 0; n < NRM; ++n)
        if (n < nR) qr[n] += dot_basis<KM>(c + n * KP, bf + t * KP);
    }
  }
#pragma unroll
  for (int n = 0; n < NRM; ++n) qr[n] = group_sum<G>(qr[n]);
  if (active && gl == 0) {
    nn_r[i] = min(cr, mn_r);
    nn_a[i] = min(ca, mn_a);
    if (heads) hrow[0] = min(ca, mn_a);
    if (cr > mn_r) atomicOr(&st->overflow, 2);
    if (ca > mn_a) atomicOr(&st->overflow, 4);
    atomicMax(&st->max_nn[1], cr);
    atomicMax(&st->max_nn[2], ca);
    atomicMax(&st->call_nn[0], cr);
    atomicMax(&st->call_nn[1], ca);
#pragma unroll
    for (int n = 0; n < NRM; ++n)
      if (n < nR) qrad[static_cast<size_t>(i) * nR + n] = qr[n];
  }
}

// Directed angular partial force of a center on one neighbour at
// r = (dx, dy, dz) = r_j - r_i:
//   f12 = (sum_lm B_lm Y_lm) r^ + (1/d)(I - r^r^T) sum_lm A_lm dY_lm/dr^,
//   A_lm = sum_n a[n][lm] g_n(d), B_lm = sum_n a[n][lm] g'_n(d),
// with a[n][lm] = dE/ds[n][lm] of the center (av: global memory, or with AG
// false the center's shared-memory scratch) and c its angular coefficient
// table for the pair (nA rows of the padded basis, shared memory).
// Reference find_partial_force_angular (nep.cu:890-991) with the
// accumulate_f12 ladder (nep_utilities.cuh:1240-1491) evaluated once per edge
// instead of once per (edge, n).  (Degrees 5 to 8; angular_edge_force4 below.)
template <int KM, int NAM, int LMAX, bool AG, bool FAST>
__device__ __forceinline__ float3 angular_edge_force(const ModelParams& p, const float* c,
                                                    const float* __restrict__ av, float rc,
                                                    float rcinv, float dx, float dy, float dz)
{
  constexpr int KP = (KM + 3) & ~3;
  constexpr int NLM = num_lm<LMAX>();
  const int nA = p.nA, L_max = p.L_max;
  float d, dinv;
  edge_length<FAST>(dx * dx + dy * dy + dz * dz, d, dinv);
  const float ux = dx * dinv, uy = dy * dinv, uz = dz * dinv;
  float fc, fcp;
  cutoff_fc<FAST>(rc, rcinv, d, fc, fcp);
  float fn[KP], fnp[KP];
#pragma unroll
  for (int kk = 0; kk < KP; ++kk) {
    fn[kk] = 0.0f;
    fnp[kk] = 0.0f;
  }
  radial_basis_d<KM>(p.kA, rcinv, d, fc, fcp, fn, fnp);
  // A and B as pairs of components (fma2)
  float2 A2[NLM / 2], B2[NLM / 2];
#pragma unroll
  for (int q = 0; q < NLM / 2; ++q) A2[q] = B2[q] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int n = 0; n < NAM; ++n) {
    if (n < nA) {
      const float g = dot_basis<KM>(c + n * KP, fn);
      const float gp = dot_basis<KM>(c + n * KP, fnp);
      const float2 g2 = make_float2(g, g), gp2 = make_float2(gp, gp);
      const float* an = av + n * NLM;
#pragma unroll
      for (int q = 0; q < NLM / 4; ++q) {
        const float4 a4 = AG ? __ldg(reinterpret_cast<const float4*>(an) + q)
                             : reinterpret_cast<const float4*>(an)[q];
        const float2 lo = make_float2(a4.x, a4.y), hi = make_float2(a4.z, a4.w);
        A2[2 * q] = fma2(lo, g2, A2[2 * q]);
        A2[2 * q + 1] = fma2(hi, g2, A2[2 * q + 1]);
        B2[2 * q] = fma2(lo, gp2, B2[2 * q]);
        B2[2 * q + 1] = fma2(hi, gp2, B2[2 * q + 1]);
      }
    }
  }
  float A[NLM], B[NLM];
#pragma unroll
  for (int q = 0; q < NLM / 2; ++q) {
    A[2 * q] = A2[q].x;
    A[2 * q + 1] = A2[q].y;
    B[2 * q] = B2[q].x;
    B[2 * q + 1] = B2[q].y;
  }
  // SB = sum B Y, V = sum A dY/du (u components independent)
  float zp[LMAX + 1];
  zp[0] = 1.0f;
#pragma unroll
  for (int q = 1; q <= LMAX; ++q) zp[q] = zp[q - 1] * uz;
  float SB = 0.0f, vx = 0.0f, vy = 0.0f, vz = 0.0f;
  int idx = 0;
#pragma unroll
  for (int Lq = 1; Lq <= LMAX; ++Lq) {
    if (Lq > L_max) break;
    float re0 = 1.0f, im0 = 0.0f;   // (ux + i uy)^(m-1)
#pragma unroll
    for (int m = 0; m <= Lq; ++m) {
      float dzf;
      const float zf = zpoly_any(Lq, m, zp, &dzf);
      if (m == 0) {
        SB += B[idx] * zf;
        vz += A[idx] * dzf;
        ++idx;
      } else {
        const float re = ux * re0 - uy * im0;
        const float im = ux * im0 + uy * re0;
        const float Ar = A[idx], Ai = A[idx + 1];
        SB += (B[idx] * re + B[idx + 1] * im) * zf;
        const float mzf = m * zf;
        vx += mzf * (Ar * re0 + Ai * im0);
        vy += mzf * (Ai * re0 - Ar * im0);
        vz += dzf * (Ar * re + Ai * im);
        idx += 2;
        re0 = re;
        im0 = im;
      }
    }
  }
  const float uv = ux * vx + uy * vy + uz * vz;
  return make_float3(SB * ux + (vx - uv * ux) * dinv, SB * uy + (vy - uv * uy) * dinv,
                     SB * uz + (vz - uv * uz) * dinv);
}

// The same for degrees <= 4, four components at a time: a component's A and B are
// used as soon as they are summed over n, so no array of them stays live (A and
// B whole took 48 registers; mixed-mode descriptor stage of 200k carbon 0.724
// -> 0.659 ms, FP32 about the same).  Two edges per lane at once, which read each
// moment derivative once for both, were no faster (1M carbon 3.35 against 3.33
// ms, copper with its 18 edges per atom 2.40 against 2.33).
template <int KM, int NAM, bool AG, bool FAST, bool EX>
__device__ __forceinline__ float3 angular_edge_force4(const ModelParams& p, const float2* cut,
                                                     const float* ctab,
                                                     const float* __restrict__ av,
                                                     const float4& e)
{
  constexpr int KP = (KM + 3) & ~3;
  constexpr int NLM = kNumLM;
  const int nA = EX ? NAM : p.nA;
  const int nlm = EX ? NLM : (p.L_max + 1) * (p.L_max + 1) - 1;
  const int t2 = row_type(e);
  const float rc = cut[t2].x, rcinv = cut[t2].y;
  float d, dinv, fc, fcp;
  edge_length<FAST>(e.x * e.x + e.y * e.y + e.z * e.z, d, dinv);
  const float ux = e.x * dinv, uy = e.y * dinv, uz = e.z * dinv;
  cutoff_fc<FAST>(rc, rcinv, d, fc, fcp);
  float2 g[NAM], gp[NAM];   // g_n, g'_n in both halves of a pair
  {
    float fn[KP], fnp[KP];
#pragma unroll
    for (int kk = 0; kk < KP; ++kk) fn[kk] = fnp[kk] = 0.0f;
    radial_basis_d<KM>(p.kA, rcinv, d, fc, fcp, fn, fnp);
    const float* c = ctab + t2 * nA * KP;
#pragma unroll
    for (int n = 0; n < NAM; ++n) {
      if (n < nA) {
        const float gn = dot_basis<KM>(c + n * KP, fn), gpn = dot_basis<KM>(c + n * KP, fnp);
        g[n] = make_float2(gn, gn);
        gp[n] = make_float2(gpn, gpn);
      }
    }
  }
  // powers of u_z and of u_x + i u_y
  float zp[5], re[5], im[5];
  zp[0] = re[0] = 1.0f;
  im[0] = 0.0f;
#pragma unroll
  for (int m = 1; m < 5; ++m) {
    zp[m] = zp[m - 1] * uz;
    re[m] = ux * re[m - 1] - uy * im[m - 1];
    im[m] = ux * im[m - 1] + uy * re[m - 1];
  }
  float SB = 0.0f, vx = 0.0f, vy = 0.0f, vz = 0.0f;
  float A[NLM], B[NLM];
#pragma unroll
  for (int q = 0; q < NLM / 4; ++q) {
    if (!EX && 4 * q >= nlm) break;
    float2 a2[2], b2[2];
    a2[0] = a2[1] = b2[0] = b2[1] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int n = 0; n < NAM; ++n) {
      if (n < nA) {
        const float4* an = reinterpret_cast<const float4*>(av + n * NLM) + q;
        const float4 a4 = AG ? __ldg(an) : *an;
        const float2 lo = make_float2(a4.x, a4.y), hi = make_float2(a4.z, a4.w);
        a2[0] = fma2(lo, g[n], a2[0]);
        a2[1] = fma2(hi, g[n], a2[1]);
        b2[0] = fma2(lo, gp[n], b2[0]);
        b2[1] = fma2(hi, gp[n], b2[1]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      A[4 * q + 2 * h] = a2[h].x;
      A[4 * q + 2 * h + 1] = a2[h].y;
      B[4 * q + 2 * h] = b2[h].x;
      B[4 * q + 2 * h + 1] = b2[h].y;
    }
    // the components whose (re, im) pair ends in this four
    int idx = 0;
#pragma unroll
    for (int L = 1; L <= 4; ++L) {
#pragma unroll
      for (int m = 0; m <= L; ++m) {
        const int last = m == 0 ? idx : idx + 1;
        if (last / 4 == q) {
          float dzf;
          const float zf = zpoly(L, m, zp, &dzf);
          if (m == 0) {
            SB += B[idx] * zf;
            vz += A[idx] * dzf;
          } else {
            const float Ar = A[idx], Ai = A[idx + 1];
            const float mzf = m * zf;
            SB += (B[idx] * re[m] + B[idx + 1] * im[m]) * zf;
            vx += mzf * (Ar * re[m - 1] + Ai * im[m - 1]);
            vy += mzf * (Ai * re[m - 1] - Ar * im[m - 1]);
            vz += dzf * (Ar * re[m] + Ai * im[m]);
          }
        }
        idx = last + 1;
      }
    }
  }
  const float uv = ux * vx + uy * vy + uz * vz;
  return make_float3(SB * ux + (vx - uv * ux) * dinv, SB * uy + (vy - uv * uy) * dinv,
                     SB * uz + (vz - uv * uz) * dinv);
}

// (cut: the center's type's row of the angular pair cutoffs, ctab of the tables.)
// Forces of the edges erow[0 .. na) of one center into frow (which may be the
// same memory: each lane reads an edge before it writes the force), by the G
// lanes of a group, the next edge loaded one iteration early.
template <int G, int KM, int NAM, int LMAX, bool AG, bool FAST, bool EX>
__device__ __forceinline__ void angular_force_row(const ModelParams& p, const float2* cut,
                                                  const float* ctab,
                                                  const float* __restrict__ av, int na, int gl,
                                                  const float4* erow, float4* frow)
{
  float4 next = make_float4(1.0f, 0.0f, 0.0f, 0.0f);
  if (gl < na) next = erow[gl];
  for (int k = gl; k < na; k += G) {
    const float4 e = next;
    if (k + G < na) next = erow[k + G];
    float3 f;
    if constexpr (LMAX <= 4) {
      f = angular_edge_force4<KM, NAM, AG, FAST, EX>(p, cut, ctab, av, e);
    } else {
      const int t2 = row_type(e);
      f = angular_edge_force<KM, NAM, LMAX, AG, FAST>(
        p, ctab + t2 * p.nA * ((KM + 3) & ~3), av, cut[t2].x, cut[t2].y, e.x, e.y, e.z);
    }
    frow[k] = make_float4(f.x, f.y, f.z, 0.0f);
  }
}

// NRM/KM/NAM: compile-time bounds of nR, basis size + 1, nA for this instance.
// MINB: CTAs per SM the instance is built for (register cap 65536 / (128
// MINB)).  The small shape comes at 3 (168 registers, moments of five radial
// functions per sweep) and at 4 (128 registers, three per sweep: the angular
// row is swept twice but a third more warps hide the latency); the
// autotuner picks one.
// XR: explicit rows (small-box and batched paths) -- the radial and angular
// rows hold the displacement and packed neighbour of every edge (er, ea),
// built beforehand; phase 1 then only accumulates the radial descriptors.
// LMAX: 4 (moments of 24 components per n, five n per sweep) or 8 (80
// components, one n per sweep).
// TC: the ANN of the CTA's centers runs on the tensor cores (tc_ann, the
// mixed-precision path); otherwise in FP32 per center.
// FF (Verlet-row path only): the kernel ends with the directed angular partial
// forces f12 of the center's edges, from a[n][lm] in its shared-memory
// scratch, in place of handing a[n][lm] to k_angular_f12 through memory (the
// autotuner times both forms).
// EX: the model has exactly the instance's shape (nR = NRM, nA = NAM, both
// bases KM, L_max = LMAX), so every such bound is a compile-time constant: the
// edge loops become straight lines without a comparison per n and degree.
// With the moments and the A/B coefficients summed in packed pairs (fma2) it
// took the descriptor stage of 1M carbon from 4.59 to 4.03 ms (FP32), of 200k
// carbon in the mixed mode from 0.922 to 0.803 ms, of water 24k from 0.152 to
// 0.142 ms; the kernel issued 1,660 warp instructions per atom, from 2,190.
template <int G, int NRM, int KM, int NAM, bool XR, int LMAX, int MINB, bool TC, bool FF, bool EX>
__global__ void __launch_bounds__(kBlock, MINB)
k_nep_fused(const ModelParams p, int N, const Site* __restrict__ sites, NeighborState* st,
            const int* __restrict__ nn_r, int mn_r, const int* __restrict__ nn_a, int mn_a,
            const float4* __restrict__ er, const float4* __restrict__ ea,
            const float* __restrict__ qrad, float* __restrict__ alpha, float* __restrict__ acoef,
            float4* f12, double* __restrict__ pe_ann)
{
  static_assert(!(FF && XR), "the fused angular force is built for Verlet rows only");
  // the mixed-precision build also takes the hardware approximations of
  // sqrt, reciprocal, sine and cosine (cutoff_fc)
  constexpr bool FAST = TC;
  constexpr int APW = 32 / G;             // centers per warp
  constexpr int APB = kBlock / G;         // centers per block
  constexpr int KP = (KM + 3) & ~3;
  constexpr int NLM = num_lm<LMAX>();
  // radial functions per moment sweep
  constexpr int CN =
    LMAX <= 4 ? (MINB >= (KM <= 9 ? 4 : 3) ? kChunkN4 : kChunkN) : 1;
  extern __shared__ __align__(128) float sm[];
  const FusedLayout Lay = fused_layout(p, APB, KP, fused_smem_budget(MINB), TC);
  const int tid = threadIdx.x;
  const int T = p.T, nR = EX ? NRM : p.nR, nA = EX ? NAM : p.nA;
  const int kR = EX ? KM : p.kR, kA = EX ? KM : p.kA, L_max = EX ? LMAX : p.L_max;
  const int dim = p.dim, H = p.H;
  // padded coefficient tables
  for (int k = tid; k < T * T * nR * Lay.kpr; k += kBlock) {
    const int kk = k % Lay.kpr, row = k / Lay.kpr;   // row = tp*nR + n
    sm[Lay.c_rad + k] = kk < kR ? __ldg(p.c_pair + row * kR + kk) : 0.0f;
  }
  for (int k = tid; k < T * T * nA * Lay.kpa; k += kBlock) {
    const int kk = k % Lay.kpa, row = k / Lay.kpa;
    sm[Lay.c_ang + k] = kk < kA ? __ldg(p.c_pair + p.num_c_radial + row * kA + kk) : 0.0f;
  }
  float2* cut_r = reinterpret_cast<float2*>(sm + Lay.cut_r);
  float2* cut_a = reinterpret_cast<float2*>(sm + Lay.cut_a);
  load_pair_cut(p, 0, cut_r);
  load_pair_cut(p, 1, cut_a);
  if (Lay.wt >= 0) {
    const float4* src = reinterpret_cast<const float4*>(p.w0t);
    float4* dst = reinterpret_cast<float4*>(sm + Lay.wt);
    for (int k = tid; k < T * dim * p.H4 / 4; k += kBlock) dst[k] = __ldg(src + k);
  }
  if (blockIdx.x == 0 && tid == 0) st->rebuild = 0;   // the Verlet list is consumed
  if constexpr (TC) {
    tc_ann_setup<APB>(p, Lay, reinterpret_cast<unsigned char*>(sm));
    tc::before_sync();
  }
  __syncthreads();
  if constexpr (TC) tc::after_sync();

  const int lane = tid & 31, warp = tid >> 5;
  const int group = lane / G, gl = lane % G;
  const int slot = warp * APW + group;                 // center within the block
  const int i = blockIdx.x * APB + slot;
  const bool active = i < N;
  float* mine = sm + Lay.atoms_base + slot * Lay.per_atom;
  float* s_s = mine + Lay.s;
  float* s_a = mine + Lay.a;
  float* s_q = mine + Lay.q;
  float* s_fp = mine + Lay.fp;
  const int t1 = active ? static_cast<int>(sites[i].type) : 0;

  // ---- 1. filter the Verlet row, radial descriptors -------------------------
  float qr[NRM];
#pragma unroll
  for (int n = 0; n < NRM; ++n) qr[n] = 0.0f;
  // q_n += sum_k c(t1,t2)[n][k] f_k(d) for one radial edge
  auto add_radial = [&](int t2, float d12_square) {
    const float rc_radial = cut_r[t1 * T + t2].x, rcinv = cut_r[t1 * T + t2].y;
    float d, dinv;
    edge_length<FAST>(d12_square, d, dinv);
    float fc, fcp;
    cutoff_fc<FAST>(rc_radial, rcinv, d, fc, fcp);
    float fn[KP];
#pragma unroll
    for (int kk = 0; kk < KP; ++kk) fn[kk] = 0.0f;
    radial_basis<KM>(kR, rcinv, d, fc, fn);
    const float* c = sm + Lay.c_rad + (t1 * T + t2) * nR * Lay.kpr;
#pragma unroll
    for (int n = 0; n < NRM; ++n)
      if (n < nR) qr[n] += dot_basis<KM>(c + n * Lay.kpr, fn);
  };
  int cr = 0, ca = 0;
  if constexpr (XR) {
    // explicit rows: counts clamped to capacity by the row builder
    cr = active ? nn_r[i] : 0;
    ca = active ? nn_a[i] : 0;
    const int cr_max = __reduce_max_sync(kFull, cr);
    const float4* erow = er + static_cast<size_t>(i) * mn_r;
    for (int base = 0; base < cr_max; base += G) {
      const int k = base + gl;
      if (k < cr) {
        const float4 e = erow[k];
        const int t2 = row_type(e);
        add_radial(t2, e.x * e.x + e.y * e.y + e.z * e.z);
      }
    }
  } else {
    // the typewise rows, their counts and the radial descriptors come from
    // k_filter_radial (lane 0 of the group holds q, the group sum spreads it)
    cr = active ? nn_r[i] : 0;
    ca = active ? nn_a[i] : 0;
    if (active && gl == 0)
#pragma unroll
      for (int n = 0; n < NRM; ++n)
        if (n < nR) qr[n] = qrad[static_cast<size_t>(i) * nR + n];
  }
#pragma unroll
  for (int n = 0; n < NRM; ++n) qr[n] = group_sum<G>(qr[n]);
  if (gl == 0)
#pragma unroll
    for (int n = 0; n < NRM; ++n)
      if (n < nR) s_q[n] = qr[n];
  __syncwarp();

  // ---- 2. angular moments s[n][lm] -----------------------------------------
  const int na = min(ca, mn_a);
  const int na_max = __reduce_max_sync(kFull, na);
  // the angular edges (displacement, neighbour type): the explicit row, or
  // what k_filter_radial left in the slots of the forces; the next edge is
  // loaded one iteration early
  const float4* earow = (XR ? ea : f12) + static_cast<size_t>(i) * mn_a;
  for (int nc = 0; nc < nA; nc += CN) {
    // padded to a whole share per lane
    constexpr int VL = (CN * NLM + G - 1) / G * G;
    float v[VL];
#pragma unroll
    for (int q = 0; q < VL; ++q) v[q] = 0.0f;
    float4 e_next = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (gl < na) e_next = earow[gl];
    for (int base = 0; base < na_max; base += G) {
      const int k = base + gl;
      const float4 e = e_next;
      if (k + G < na) e_next = earow[k + G];
      if (k < na) {
        const float dx = e.x, dy = e.y, dz = e.z;
        const int t2 = row_type(e);
        float d, dinv;
        edge_length<FAST>(dx * dx + dy * dy + dz * dz, d, dinv);
        const float2 cut = cut_a[t1 * T + t2];
        const float rc = cut.x, rcinv = cut.y;
        float fc, fcp;
        cutoff_fc<FAST>(rc, rcinv, d, fc, fcp);
        float fn[KP];
#pragma unroll
        for (int kk = 0; kk < KP; ++kk) fn[kk] = 0.0f;
        radial_basis<KM>(kA, rcinv, d, fc, fn);
        const float* c = sm + Lay.c_ang + ((t1 * T + t2) * nA + nc) * Lay.kpa;
        float g[CN];
#pragma unroll
        for (int n = 0; n < CN; ++n)
          g[n] = (nc + n < nA) ? dot_basis<KM>(c + n * Lay.kpa, fn) : 0.0f;
        // components two at a time (fma2): an even one waits for the odd one after it
        float even = 0.0f;
        for_each_harmonic<LMAX>(L_max, dx * dinv, dy * dinv, dz * dinv, [&](int lm, float y) {
          if ((lm & 1) == 0) {
            even = y;
            return;
          }
#pragma unroll
          for (int n = 0; n < CN; ++n) {
            float* w = v + n * NLM + lm - 1;
            const float2 r = fma2(make_float2(even, y), make_float2(g[n], g[n]),
                                  make_float2(w[0], w[1]));
            w[0] = r.x;
            w[1] = r.y;
          }
        });
        if constexpr (!EX) {
          // an odd L_max ends on an even component
#pragma unroll
          for (int L = 1; L <= LMAX; L += 2)
            if (L == L_max)
#pragma unroll
              for (int n = 0; n < CN; ++n) v[n * NLM + L * L + 2 * L - 1] += g[n] * even;
        }
      }
    }
    const int at = reduce_scatter<G, VL>(v, gl);
    constexpr int share = VL / G;
    const int lim = (nA - nc < CN ? nA - nc : CN) * NLM;
#pragma unroll
    for (int q = 0; q < share; ++q)
      if (at + q < lim) s_s[nc * NLM + at + q] = v[q];
  }
  __syncwarp();

  // ---- 3. invariants, ANN, derivatives ---------------------------------------
  if constexpr (NLM == kNumLM) {
    // degrees <= 4: the n's 24 moments in registers, monomials unrolled
    for (int n = gl; n < nA; n += G) {
      float sv[kNumLM];
      load24(s_s + n * NLM, sv);
      float* q = s_q + nR;
#pragma unroll
      for (int Lq = 1; Lq <= 4; ++Lq) {
        if (Lq <= L_max) {
          const int st0 = Lq * Lq - 1;
          float val = 0.0f;
#pragma unroll
          for (int k = 1; k < 2 * Lq + 1; ++k) val += c_C3B[st0 + k] * sv[st0 + k] * sv[st0 + k];
          val *= 2.0f;
          val += c_C3B[st0] * sv[st0] * sv[st0];
          q[(Lq - 1) * nA + n] = val;
        }
      }
      int col = L_max;
      for (int w = 0; w < p.num_inv; ++w, ++col) q[col * nA + n] = inv_value_id(p.inv_id[w], sv);
    }
  } else {
    for (int n = gl; n < nA; n += G) {
      const float* s = s_s + n * NLM;
      float* q = s_q + nR;
      int col = 0;
      for (int Lq = 1; Lq <= L_max; ++Lq, ++col) {
        const int st0 = Lq * Lq - 1;
        float val = 0.0f;
        for (int k = 1; k < 2 * Lq + 1; ++k) val += c_C3B[st0 + k] * s[st0 + k] * s[st0 + k];
        val *= 2.0f;
        val += c_C3B[st0] * s[st0] * s[st0];
        q[col * nA + n] = val;
      }
      for (int w = 0; w < p.num_inv; ++w, ++col) {
        const int id = p.inv_id[w];
        float acc = 0.0f;
        for (int m = c_inv_start[id]; m < c_inv_start[id + 1]; ++m) {
          const Monomial mo = c_mono[m];
          float t = mo.c * s[mo.i[0]] * s[mo.i[1]] * s[mo.i[2]];
          if (mo.i[3] >= 0) t *= s[mo.i[3]];
          acc += t;
        }
        q[col * nA + n] = acc;
      }
    }
  }
  __syncwarp();
  // scaled descriptors; hidden-unit derivatives zero-padded to H4 for the
  // float4 dot products
  for (int d = gl; d < dim; d += G) s_q[d] *= __ldg(p.q_scaler + d);
  if constexpr (TC) {
    __syncwarp();
    tc_ann<APB, G>(p, Lay, sm, slot, gl, active, t1, i, s_q, pe_ann, st);
  } else {
    // In this stage adjacent lanes take different centers of the warp and the
    // same hidden units (ag: this lane's share of them): a 16-byte read of the
    // weights is then the same for the lanes of one type, which costs the
    // shared-memory pipe 2.3 cycles, where four lanes of a center with four
    // rows each took 4 (forward) and, at the rows' common bank, 8 (backward).
    const int ac = lane % APW, ag = lane / APW;
    const int a_slot = warp * APW + ac, a_i = blockIdx.x * APB + a_slot;
    const bool a_active = a_i < N;
    const int a_t = __shfl_sync(kFull, t1, ac * G);
    float* a_mine = sm + Lay.atoms_base + a_slot * Lay.per_atom;
    const float* a_q = a_mine + Lay.q;
    float* a_fp = a_mine + Lay.fp;
    float* a_gh = a_mine + Lay.gh;
    for (int h = H + ag; h < p.H4; h += G) a_gh[h] = 0.0f;
    __syncwarp();
    const float* w0t = Lay.wt >= 0 ? sm + Lay.wt : p.w0t;
    const int hq = p.H4 / 4;
    const float4* wt = reinterpret_cast<const float4*>(w0t + static_cast<size_t>(a_t) * dim * p.H4);
    float e_part = 0.0f;
    if (a_active) {
      // hidden layer: each lane owns two groups of four consecutive hidden units
      // (float4 rows of the transposed w0; four chains of packed pairs in one
      // pass, each sequential in d as in the reference)
      auto finish = [&](int h, float z) {
        if (h < H) {
          const float x1 = tanhf(z - __ldg(p.b0 + a_t * H + h));
          const float w1 = __ldg(p.w1 + a_t * H + h);
          e_part += w1 * x1;
          a_gh[h] = w1 * (1.0f - x1 * x1);
        }
      };
      for (int h4 = ag; h4 < hq; h4 += 2 * G) {
        const bool has_b = h4 + G < hq;
        const int h4b = has_b ? h4 + G : h4;   // past the end: computed, dropped
        float2 z01 = make_float2(0.0f, 0.0f), z23 = z01, z45 = z01, z67 = z01;
#pragma unroll 4
        for (int d = 0; d < dim; ++d) {
          const float q = a_q[d];
          const float2 q2 = make_float2(q, q);
          const float4 wa = wt[d * hq + h4];
          const float4 wb = wt[d * hq + h4b];
          z01 = fma2(make_float2(wa.x, wa.y), q2, z01);
          z23 = fma2(make_float2(wa.z, wa.w), q2, z23);
          z45 = fma2(make_float2(wb.x, wb.y), q2, z45);
          z67 = fma2(make_float2(wb.z, wb.w), q2, z67);
        }
        finish(4 * h4, z01.x);
        finish(4 * h4 + 1, z01.y);
        finish(4 * h4 + 2, z23.x);
        finish(4 * h4 + 3, z23.y);
        if (has_b) {
          finish(4 * h4b, z45.x);
          finish(4 * h4b + 1, z45.y);
          finish(4 * h4b + 2, z67.x);
          finish(4 * h4b + 3, z67.y);
        }
      }
    }
#pragma unroll
    for (int o = APW; o < 32; o <<= 1) e_part += __shfl_xor_sync(kFull, e_part, o);
    if (a_active && ag == 0) pe_ann[a_i] = static_cast<double>(e_part - __ldg(p.out_bias + a_t));
    __syncwarp();
    if (a_active) {
      // dE/dq: four descriptor components per lane at once (d0, d0 + G,
      // d0 + 2G, d0 + 3G), float4 over h, even and odd hidden units apart
      const float4* g4 = reinterpret_cast<const float4*>(a_gh);
      for (int d0 = ag; d0 < dim; d0 += 4 * G) {
        int dd[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) dd[k] = min(d0 + k * G, dim - 1);   // past dim: dropped
        float2 acc[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = make_float2(0.0f, 0.0f);
#pragma unroll 2
        for (int h = 0; h < hq; ++h) {
          const float4 g = g4[h];
          const float2 g01 = make_float2(g.x, g.y), g23 = make_float2(g.z, g.w);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 w = wt[dd[k] * hq + h];
            acc[k] = fma2(g01, make_float2(w.x, w.y), acc[k]);
            acc[k] = fma2(g23, make_float2(w.z, w.w), acc[k]);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (d0 + k * G < dim)
            a_fp[d0 + k * G] = (acc[k].x + acc[k].y) * __ldg(p.q_scaler + d0 + k * G);
      }
    }
    __syncwarp();
  }
  if (active) center_alpha<G>(T, nR, t1, s_fp, sm + Lay.c_rad, Lay.kpr,
                              alpha_row<KM>(), gl,
                              alpha + static_cast<size_t>(i) * T * alpha_row<KM>());
  center_acoef<G, NLM>(p, nR, nA, L_max, s_s, s_a, s_fp, gl);
  __syncwarp();

  // ---- 4. hand a[n][lm] to the angular-force kernel -------------------------
  if constexpr (!FF) {
    if (active) {
      float4* dst = reinterpret_cast<float4*>(acoef + static_cast<size_t>(i) * nA * NLM);
      const float4* src = reinterpret_cast<const float4*>(s_a);
      for (int q = gl; q < nA * NLM / 4; q += G) dst[q] = src[q];
    }
  } else {
    // ---- 4'. or evaluate the angular partial forces here (k_angular_f12's
    // arithmetic, the moment derivatives read from shared memory), each in the
    // place of its edge
    const float* ctab = sm + Lay.c_ang + t1 * T * nA * Lay.kpa;
    float4* frow = f12 + static_cast<size_t>(i) * mn_a;
    angular_force_row<G, KM, NAM, LMAX, false, FAST, EX>(p, cut_a + t1 * T, ctab, s_a, na, gl, frow,
                                                         frow);
  }
}

// Angular coefficient tables [T*T][nA][KP] into shared memory (zero-padded rows),
// and behind them the angular pair cutoffs.
__host__ __device__ inline int angular_table_floats(const ModelParams& p, int kp)
{
  return p.T * p.T * (p.nA * kp + 2);
}
template <int KP>
__device__ __forceinline__ void load_angular_tables(const ModelParams& p, float* sm)
{
  load_pair_cut(p, 1, reinterpret_cast<float2*>(sm + p.T * p.T * p.nA * KP));
  const int T = p.T, nA = p.nA, kA = p.kA;
  for (int k = threadIdx.x; k < T * T * nA * KP; k += blockDim.x) {
    const int kk = k % KP, row = k / KP;
    sm[k] = kk < kA ? __ldg(p.c_pair + p.num_c_radial + row * kA + kk) : 0.0f;
  }
}

// One group of G lanes per center: the directed angular partial force of
// every edge of the center's angular row, f12[i][k] (float4, w unused).
// XR: explicit rows of a batch; only the centers of structures that are not
// small (each neighbour once in their rows) take this scheme.
// FAST builds held to four CTAs per SM (128 registers, as the exact build
// takes; they would take 142, rounded to 144: three CTAs).
template <int G, int KM, int NAM, bool XR, int LMAX, bool FAST>
__global__ void __launch_bounds__(kBlock, (FAST ? 4 : 0))
k_angular_f12(const ModelParams p, int N, const Site* __restrict__ sites,
              const int* __restrict__ nn_a, int mn_a, const float4* __restrict__ ea,
              const unsigned char* __restrict__ large, const float* __restrict__ acoef,
              float4* f12)
{
  constexpr int KP = (KM + 3) & ~3;
  extern __shared__ float sm[];
  load_angular_tables<KP>(p, sm);
  __syncthreads();
  const int tid = threadIdx.x;
  const int T = p.T, nA = p.nA;
  const int gl = tid % G;
  const int i = blockIdx.x * (kBlock / G) + tid / G;
  if (i >= N) return;
  if constexpr (XR) {
    if (!large[i]) return;
  }
  const int t1 = static_cast<int>(sites[i].type);
  const int na = nn_a[i];
  const float* ai = acoef + static_cast<size_t>(i) * nA * num_lm<LMAX>();
  float4* frow = f12 + static_cast<size_t>(i) * mn_a;
  // Verlet rows: k_filter_radial left the edge in the slot of its force
  const float4* erow = XR ? ea + static_cast<size_t>(i) * mn_a : frow;
  const float2* cut = reinterpret_cast<const float2*>(sm + T * T * nA * KP) + t1 * T;
  angular_force_row<G, KM, NAM, LMAX, true, FAST, false>(p, cut, sm + t1 * T * nA * KP, ai, na,
                                                         gl, erow, frow);
}

// ---------------------------------------------------------------------------
// gather
// ---------------------------------------------------------------------------

// Eight consecutive 32-bit entries (32-byte aligned) in one load.
__device__ __forceinline__ void load8(const int* __restrict__ at, int (&v)[8])
{
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "l"(at));
}

// The rows of heads from finished angular rows, a thread per slot (the filter
// writes them on its way, except where they share the memory of its Verlet rows).
__global__ void __launch_bounds__(256)
k_row_heads(int N, const int* __restrict__ nn_a, const int* __restrict__ nl_a, int st_a,
            int* __restrict__ heads, int st_h)
{
  const int slots = 1 + st_a / 8;
  const long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int i = static_cast<int>(k / slots), q = static_cast<int>(k % slots);
  if (i >= N) return;
  const int n = nn_a[i];
  if (q == 0) heads[static_cast<size_t>(i) * st_h] = n;
  else if (8 * (q - 1) < n)
    heads[static_cast<size_t>(i) * st_h + q] = nl_a[static_cast<size_t>(i) * st_a + 8 * (q - 1)];
}

// Slot of atom i in an ascending row, -1 if it is not there (a truncated row):
// the last block of eight whose head is not above i, from the row of heads (the
// row's length, then its every eighth entry), then the place in that block.  Two
// rounds of loads that each wait for the one before; a binary search of a carbon
// row (34 entries) takes seven with the length, of 11 cycles of the load pipe each,
// and the gather is bound by that pipe (75 % busy).
__device__ __forceinline__ int reverse_slot(const int* __restrict__ row,
                                            const int* __restrict__ heads, int i)
{
  int v[8];
  load8(heads, v);
  const int count = v[0];
  int block = -1;
#pragma unroll
  for (int q = 1; q < 8; ++q)
    if (8 * (q - 1) < count && v[q] <= i) block = q - 1;
  for (int h0 = 8; 8 * (h0 - 1) < count; h0 += 8) {   // rows above 56 entries
    load8(heads + h0, v);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (8 * (h0 + q - 1) < count && v[q] <= i) block = h0 + q - 1;
  }
  if (block < 0) return -1;
  int slot = -1;
  load8(row + 8 * block, v);
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (8 * block + q < count && v[q] == i) slot = 8 * block + q;
  return slot;
}

// ROWS: kVerlet; kImages, explicit rows that may hold one neighbour several
// times (periodic images), so the reverse partial force f12(j,i) is not looked up
// but evaluated here from j's moment derivatives at -r (the angular force work
// doubles and the f12 buffer and its kernel drop out); kLarge, the explicit rows
// of a batch's structures that are not small, which hold each neighbour once and
// take the Verlet rows' scheme.  A batch launches both explicit builds, each over
// its own centers: one build for both took 103 registers and two CTAs per SM for
// the centers that need neither angular force.
// GMINB: CTAs of 256 per SM the instance is built for (register cap), 0 for
// none.  The Verlet-row gather comes uncapped (74 registers for the small shape,
// three CTAs) and at 4 (64 registers, a third more warps); the autotuner picks
// one.  The small shape's FAST build of kImages is held to two CTAs.
constexpr int kVerlet = 0, kImages = 1, kLarge = 2;
template <int G, int KM, int NAM, int ROWS, int LMAX, int GMINB, bool FAST>
__global__ void __launch_bounds__(256, GMINB)
k_gather(const ModelParams p, int N, const Box* __restrict__ box,
         const Site* __restrict__ sites, const int* __restrict__ nn_r, const int* __restrict__ nl_r,
         int mn_r, const int* __restrict__ nn_a, const int* __restrict__ nl_a, int mn_a, int st_a,
         const int* __restrict__ heads, int st_h, const float4* __restrict__ er, const float4* __restrict__ ea,
         const float* __restrict__ acoef, const float* __restrict__ alpha,
         const float4* __restrict__ f12, const unsigned char* __restrict__ large,
         const double* __restrict__ pe_ann,
         double* __restrict__ pe, double* __restrict__ force, double* __restrict__ virial,
         int accumulate, NeighborState* st)
{
  constexpr int KP = (KM + 3) & ~3;
  constexpr bool XR = ROWS != kVerlet, IMG = ROWS == kImages;
  extern __shared__ float sm[];
  // radial pair cutoffs, the box's matrix, (explicit rows) the angular tables
  const int T = p.T;
  float2* cut_r = reinterpret_cast<float2*>(sm);
  float* s_fh = sm + 2 * T * T;
  float* s_ang = s_fh + 18 + (2 * T * T + 18) % 4;
  load_pair_cut(p, 0, cut_r);
  const MinImage mic(box, s_fh);
  if constexpr (IMG) load_angular_tables<KP>(p, s_ang);
  __syncthreads();
  const float2* cut_a = reinterpret_cast<const float2*>(s_ang + T * T * p.nA * KP);   // IMG
  const int gl = threadIdx.x % G;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  bool active = i < N;
  if constexpr (XR) active = active && (large[i] != 0) == (ROWS == kLarge);
  const int kR = p.kR;
  constexpr int AR = alpha_row<KM>();
  float F[3] = {0.0f, 0.0f, 0.0f};
  float W[9] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  float ezbl = 0.0f;
  if (active) {
    const Site me = sites[i];
    const double xi = me.x, yi = me.y, zi = me.z;
    const int t1 = static_cast<int>(me.type);
    const float* ali = alpha + static_cast<size_t>(i) * T * AR;
    // radial pairs: both site energies through the alpha coefficients
    const int nr = nn_r[i];
    const int* rrow = nl_r + static_cast<size_t>(i) * mn_r;
    // the next edge's index is loaded one iteration early: the site and alpha
    // loads of an edge then issue together at the top of its iteration
    int jr_next = (!XR && gl < nr) ? rrow[gl] : 0;
    for (int k = gl; k < nr; k += G) {
      int j, t2;
      float dx, dy, dz;
      const int jr = jr_next;
      if constexpr (!XR) {
        if (k + G < nr) jr_next = rrow[k + G];
      }
      if constexpr (XR) {
        const float4 e = er[static_cast<size_t>(i) * mn_r + k];
        const unsigned bits = static_cast<unsigned>(__float_as_int(e.w));
        j = static_cast<int>(bits & kRowIndexMask);
        t2 = static_cast<int>(bits >> kRowTypeShift);
        dx = e.x;
        dy = e.y;
        dz = e.z;
      } else {
        j = jr;
        double2 sa, sc;
        site_load(sites, j, sa, sc);
        site_delta(mic, sa, sc, xi, yi, zi, dx, dy, dz, t2);
      }
      float d, dinv;
      edge_length<FAST>(dx * dx + dy * dy + dz * dz, d, dinv);
      const float rc = cut_r[t1 * T + t2].x, rcinv = cut_r[t1 * T + t2].y;
      float fc, fcp;
      cutoff_fc<FAST>(rc, rcinv, d, fc, fcp);
      float fn[KP], fnp[KP];
#pragma unroll
      for (int kk = 0; kk < KP; ++kk) {
        fn[kk] = 0.0f;
        fnp[kk] = 0.0f;
      }
      radial_basis_d<KM>(kR, rcinv, d, fc, fcp, fn, fnp);
      const float w12 = dot_alpha<KM>(ali + t2 * AR, fnp);
      const float w21 = dot_alpha<KM>(alpha + (static_cast<size_t>(j) * T + t1) * AR, fnp);
      const float s12 = w12 * dinv, s21 = w21 * dinv;
      // f12 = s12 r, f21 = -s21 r; F += f12 - f21; W += r (x) f21
      F[0] += (s12 + s21) * dx;
      F[1] += (s12 + s21) * dy;
      F[2] += (s12 + s21) * dz;
      const float f21[3] = {-s21 * dx, -s21 * dy, -s21 * dz};
      W[0] += dx * f21[0];
      W[1] += dy * f21[1];
      W[2] += dz * f21[2];
      W[3] += dx * f21[1];
      W[4] += dx * f21[2];
      W[5] += dy * f21[2];
    }
    // a radial pair force lies along its edge: its virial is symmetric
    W[6] = W[3];
    W[7] = W[4];
    W[8] = W[5];
    // angular exchange and ZBL
    const int na = nn_a[i];
    const int* arow = nl_a + static_cast<size_t>(i) * st_a;
    const int zi_ = p.Z[t1];
    const float pow_zi = p.zbl ? powf(static_cast<float>(zi_), 0.23f) : 0.0f;
    int ja_next = (!XR && gl < na) ? arow[gl] : 0;
    for (int k = gl; k < na; k += G) {
      int t2, rev;
      float dx, dy, dz;
      float4 a12, a21;
      const int ja = ja_next;
      if constexpr (!XR) {
        if (k + G < na) ja_next = arow[k + G];
      }
      if constexpr (XR) {
        const float4 e = ea[static_cast<size_t>(i) * mn_a + k];
        const unsigned bits = static_cast<unsigned>(__float_as_int(e.w));
        const int j = static_cast<int>(bits & kRowIndexMask);
        t2 = static_cast<int>(bits >> kRowTypeShift);
        dx = e.x;
        dy = e.y;
        dz = e.z;
        if constexpr (IMG) {
          const int nA = p.nA;
          constexpr int NLM = num_lm<LMAX>();
          const float* av_i = acoef + static_cast<size_t>(i) * nA * NLM;
          const float* av_j = acoef + static_cast<size_t>(j) * nA * NLM;
          float3 fij, fji;
          if constexpr (LMAX <= 4) {
            const float4 back =
              make_float4(-dx, -dy, -dz, __int_as_float(t1 << kRowTypeShift));
            fij = angular_edge_force4<KM, NAM, true, FAST, false>(
              p, cut_a + t1 * T, s_ang + t1 * T * nA * KP, av_i, e);
            fji = angular_edge_force4<KM, NAM, true, FAST, false>(
              p, cut_a + t2 * T, s_ang + t2 * T * nA * KP, av_j, back);
          } else {
            const float2 cut = cut_a[t1 * T + t2];
            fij = angular_edge_force<KM, NAM, LMAX, true, FAST>(
              p, s_ang + (t1 * T + t2) * nA * KP, av_i, cut.x, cut.y, dx, dy, dz);
            fji = angular_edge_force<KM, NAM, LMAX, true, FAST>(
              p, s_ang + (t2 * T + t1) * nA * KP, av_j, cut.x, cut.y, -dx, -dy, -dz);
          }
          a12 = make_float4(fij.x, fij.y, fij.z, 0.0f);
          a21 = make_float4(fji.x, fji.y, fji.z, 0.0f);
        }
        rev = j;
      } else {
        double2 sa, sc;
        site_load(sites, ja, sa, sc);
        site_delta(mic, sa, sc, xi, yi, zi, dx, dy, dz, t2);
        rev = ja;
      }
      if constexpr (!IMG) {
        a12 = f12[static_cast<size_t>(i) * mn_a + k];
        // reverse slot: i inside j's ascending row
        const int slot = reverse_slot(nl_a + static_cast<size_t>(rev) * st_a,
                                      heads + static_cast<size_t>(rev) * st_h, i);
        if (slot >= 0) {
          a21 = f12[static_cast<size_t>(rev) * mn_a + slot];
        } else {
          // only a truncated (overflowed) row can lose the reverse edge
          a21 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          atomicOr(&st->overflow, 4);
        }
      }
      F[0] += a12.x - a21.x;
      F[1] += a12.y - a21.y;
      F[2] += a12.z - a21.z;
      W[0] += dx * a21.x;
      W[1] += dy * a21.y;
      W[2] += dz * a21.z;
      W[3] += dx * a21.y;
      W[4] += dx * a21.z;
      W[5] += dy * a21.z;
      W[6] += dy * a21.x;
      W[7] += dz * a21.x;
      W[8] += dz * a21.y;
      if (p.zbl) {
        const float d = sqrtf(dx * dx + dy * dy + dz * dz);
        const float dinv = 1.0f / d;
        const int zj = p.Z[t2];
        const float a_inv = (pow_zi + powf(static_cast<float>(zj), 0.23f)) * 2.134563f;
        const float zizj = kCoulomb * zi_ * zj;
        float f, fpz;
        if (p.zbl_flexible) {
          const int ta = min(t1, t2), tb = max(t1, t2);
          const int idx = ta * p.T - (ta * (ta - 1)) / 2 + (tb - ta);
          float zpar[10];
#pragma unroll
          for (int q = 0; q < 10; ++q) zpar[q] = __ldg(p.zbl_para + 10 * idx + q);
          zbl_flexible(zpar, zizj, a_inv, d, dinv, f, fpz);
        } else {
          float r1 = p.zbl_rc_inner, r2 = p.zbl_rc_outer;
          if (p.typewise_zbl) {
            r2 = fminf((c_covalent[zi_ - 1] + c_covalent[zj - 1]) * p.typewise_factor, r2);
            r1 = 0.0f;
          }
          zbl_universal(zizj, a_inv, r1, r2, d, dinv, f, fpz);
        }
        const float f2 = fpz * dinv * 0.5f;
        const float h12[3] = {dx * f2, dy * f2, dz * f2};
        F[0] += 2.0f * h12[0];
        F[1] += 2.0f * h12[1];
        F[2] += 2.0f * h12[2];
        W[0] -= dx * h12[0];
        W[1] -= dy * h12[1];
        W[2] -= dz * h12[2];
        W[3] -= dx * h12[1];
        W[4] -= dx * h12[2];
        W[5] -= dy * h12[2];
        W[6] -= dy * h12[0];
        W[7] -= dz * h12[0];
        W[8] -= dz * h12[1];
        ezbl += 0.5f * f;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) F[c] = group_sum<G>(F[c]);
#pragma unroll
  for (int c = 0; c < 9; ++c) W[c] = group_sum<G>(W[c]);
  ezbl = group_sum<G>(ezbl);
  if (active && gl == 0) {
    const double e = pe_ann[i] + static_cast<double>(ezbl);
    const bool finite = isfinite(e) && isfinite(F[0]) && isfinite(F[1]) && isfinite(F[2]);
    if (accumulate) {
      pe[i] += e;
      for (int c = 0; c < 3; ++c) force[static_cast<size_t>(c) * N + i] += F[c];
      for (int c = 0; c < 9; ++c) virial[static_cast<size_t>(c) * N + i] += W[c];
    } else {
      pe[i] = e;
      for (int c = 0; c < 3; ++c) force[static_cast<size_t>(c) * N + i] = F[c];
      for (int c = 0; c < 9; ++c) virial[static_cast<size_t>(c) * N + i] = W[c];
    }
    if (!finite) st->nonfinite = 1;
  }
}

// shape classes: small (n_max <= 4, basis_size <= 8) and general
constexpr int kSmallN = 5, kSmallK = 9;
// Models with l_max 5..8 run one general-shape instance of each kernel (LMAX
// 8): their moments take 80 floats per n, so the descriptor and a-coefficient
// kernels take 16 centers per CTA (groups of 8 lanes), the force kernels 4.
constexpr int kHighFusedGroup = 8, kHighGroup = 4;

bool high_degree(const ModelParams& p) { return p.L_max > 4; }

// every kernel of a model uses one basis stride, so high-degree models take
// the general shape throughout
bool small_shape(const ModelParams& p)
{
  return !high_degree(p) && p.nR <= kSmallN && p.nA <= kSmallN && p.kR <= kSmallK &&
         p.kA <= kSmallK;
}

// The model has the small instances' exact shape (n_max 4 4, basis 8 8, l_max
// 4: the format's usual one), which has builds of its own.
bool exact_shape(const ModelParams& p)
{
  return p.nR == kSmallN && p.nA == kSmallN && p.kR == kSmallK && p.kA == kSmallK && p.L_max == 4;
}

// Builds of the exact shape: everywhere the model has it, except at four CTAs per SM
// with the angular force inside. At 128 registers the straight-line form spills 192
// bytes there, the general one of the same bounds none (force call of 24,000 water
// atoms in that build: 196 -> 182 us at 4 lanes, 182 -> 173 at 8; the three-CTA
// build takes 171).
template <int KM, int LMAX, int MINB, bool FF>
constexpr bool exact_build() { return KM == kSmallK && LMAX == 4 && !(MINB == 4 && FF); }

template <int G, int NRM, int KM, int NAM, bool XR, int LMAX, int MINB, bool TC, bool FF, bool EX>
void launch_fused_tx(Engine& e, int N, cudaStream_t s)
{
  NeighborBuffers& nb = e.nbr;
  constexpr int APB = kBlock / G;
  const int blocks = (N + APB - 1) / APB;
  const size_t smem =
    fused_layout(e.params, APB, (KM + 3) & ~3, fused_smem_budget(MINB), TC).total_bytes;
  k_nep_fused<G, NRM, KM, NAM, XR, LMAX, MINB, TC, FF, EX><<<blocks, kBlock, smem, s>>>(
    e.params, N, e.scratch.sites, e.d_nstate, nb.nn_r, nb.mn_r, nb.nn_a, nb.mn_a, e.xr.er,
    e.xr.ea, e.scratch.qrad, e.scratch.alpha, e.scratch.acoef, e.scratch.f12, e.scratch.pe_ann);
}

// Groups of 16 and 32 lanes serve small systems, where a kernel's time is one
// center's chain of edges and not the chip's throughput (4,096 atoms at 8 lanes
// are 256 CTAs of 128): FP32 builds of the exact small shape, and the filter and
// gather of the small shape, chosen by size below kWideAtoms.  Elsewhere they run
// as groups of 8.
template <int G, int NRM, int KM, int NAM, bool XR, int LMAX, int MINB, bool TC, bool FF = false>
void launch_fused_t(Engine& e, int N, cudaStream_t s)
{
  if constexpr (exact_build<KM, LMAX, MINB, FF>()) {
    if (exact_shape(e.params)) {
      launch_fused_tx<G, NRM, KM, NAM, XR, LMAX, MINB, TC, FF, true>(e, N, s);
      return;
    }
  }
  launch_fused_tx<G, NRM, KM, NAM, XR, LMAX, MINB, TC, FF, false>(e, N, s);
}

// Dynamic shared memory above the default limit: the kernel is allowed all an SM
// has, once and for every handle (a limit of one model's bytes would fall below
// what another handle's model needs).
template <typename K>
void allow_smem(K kernel, size_t bytes)
{
  if (bytes > 48 * 1024)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

// The mixed precisions take the FAST builds of the filter, angular-force and
// gather kernels (and of the descriptor kernel, whose tensor-core build is
// FAST); they exist for the small shape, the others run the exact build.
inline bool fast_math(const Engine& e) { return e.precision != 0; }

template <int G, int NRM, int KM, bool FAST>
void launch_filter_tf(Engine& e, int N, cudaStream_t s)
{
  NeighborBuffers& nb = e.nbr;
  constexpr int APB = kBlock / G, KP = (KM + 3) & ~3;
  const ModelParams& p = e.params;
  const int blocks = (N + APB - 1) / APB;
  auto launch = [&](auto kernel, size_t bin_float4) {
    const size_t smem =
      sizeof(float) * (filter_table_floats(p, KP) + 4 * kBlock * bin_float4 + 4 * p.T * p.T + 20);
    allow_smem(kernel, smem);
    kernel<<<blocks, kBlock, smem, s>>>(p, N, e.d_box, e.scratch.sites, e.d_nstate, nb.nn_v,
                                        nb.nl_v, nb.mn_v, nb.nn_r, nb.nl_r, nb.mn_r, nb.nn_a,
                                        nb.nl_a, nb.mn_a, nb.st_a,
                                        nb.heads_after_filter ? nullptr : nb.heads, nb.st_h,
                                        e.scratch.f12, e.scratch.qrad);
  };
  const int bin = filter_bin<KM>(p);
  if (bin == kBinShared)
    launch(k_filter_radial<G, NRM, KM, kBinShared, FAST>, filter_bin_float4(p, KP));
  else if (bin == kBinNone) launch(k_filter_radial<G, NRM, KM, kBinNone, FAST>, 0);
  if constexpr (KM <= 9)
    if (bin == kBinRegs) launch(k_filter_radial<G, NRM, KM, kBinRegs, FAST>, 0);
}

template <int G, int NRM, int KM>
void launch_filter_t(Engine& e, int N, cudaStream_t s)
{
  if constexpr (KM == kSmallK) {
    if (fast_math(e)) {
      launch_filter_tf<G, NRM, KM, true>(e, N, s);
      return;
    }
  }
  launch_filter_tf<G, NRM, KM, false>(e, N, s);
}

template <int G, int KM, int NAM, int LMAX, bool FAST>
void launch_f12_tf(Engine& e, int N, cudaStream_t s)
{
  NeighborBuffers& nb = e.nbr;
  constexpr int APB = kBlock / G;
  const int blocks = (N + APB - 1) / APB;
  const size_t smem = sizeof(float) * angular_table_floats(e.params, (KM + 3) & ~3);
  allow_smem(k_angular_f12<G, KM, NAM, true, LMAX, FAST>, smem);
  allow_smem(k_angular_f12<G, KM, NAM, false, LMAX, FAST>, smem);
  if (e.use_xr)
    k_angular_f12<G, KM, NAM, true, LMAX, FAST><<<blocks, kBlock, smem, s>>>(
      e.params, N, e.scratch.sites, nb.nn_a, nb.mn_a, e.xr.ea, e.xr.large, e.scratch.acoef,
      e.scratch.f12);
  else
    k_angular_f12<G, KM, NAM, false, LMAX, FAST><<<blocks, kBlock, smem, s>>>(
      e.params, N, e.scratch.sites, nb.nn_a, nb.mn_a, e.xr.ea, e.xr.large, e.scratch.acoef,
      e.scratch.f12);
}

template <int G, int KM, int NAM, int LMAX>
void launch_f12_t(Engine& e, int N, cudaStream_t s)
{
  if constexpr (KM == kSmallK && LMAX == 4) {
    if (fast_math(e)) {
      launch_f12_tf<G, KM, NAM, LMAX, true>(e, N, s);
      return;
    }
  }
  launch_f12_tf<G, KM, NAM, LMAX, false>(e, N, s);
}

// FFI: the build also comes with the fused angular force (degrees <= 4)
template <int G, int NRM, int KM, int NAM, int LMAX, int MINB, bool TC, bool FFI = false>
void set_fused_smem_t(const ModelParams& p)
{
  const int bytes =
    fused_layout(p, kBlock / G, (KM + 3) & ~3, fused_smem_budget(MINB), TC).total_bytes;
  // (only the builds this model runs, and only above the default limit: the
  // calls add up in the making of a handle)
  if constexpr (KM == kSmallK && LMAX == 4) {
    if (exact_shape(p)) {
      allow_smem(k_nep_fused<G, NRM, KM, NAM, false, LMAX, MINB, TC, false, true>, bytes);
      allow_smem(k_nep_fused<G, NRM, KM, NAM, true, LMAX, MINB, TC, false, true>, bytes);
      allow_smem(k_nep_fused<G, NRM, KM, NAM, false, LMAX, MINB, TC, true,
                             exact_build<KM, LMAX, MINB, true>()>, bytes);
      return;
    }
  }
  allow_smem(k_nep_fused<G, NRM, KM, NAM, false, LMAX, MINB, TC, false, false>, bytes);
  allow_smem(k_nep_fused<G, NRM, KM, NAM, true, LMAX, MINB, TC, false, false>, bytes);
  if constexpr (FFI)
    allow_smem(k_nep_fused<G, NRM, KM, NAM, false, LMAX, MINB, TC, true, false>, bytes);
}

template <int G>
void set_fused_smem_wide(const ModelParams& p)
{
  constexpr int n = kSmallN, k = kSmallK;
  const int bytes =
    fused_layout(p, kBlock / G, (k + 3) & ~3, fused_smem_budget(3), false).total_bytes;
  if (!exact_shape(p)) return;
  allow_smem(k_nep_fused<G, n, k, n, true, 4, 3, false, false, true>, bytes);
  allow_smem(k_nep_fused<G, n, k, n, false, 4, 3, false, true, true>, bytes);
  allow_smem(k_nep_fused<G, n, k, n, false, 4, 3, false, false, true>, bytes);
}

template <int G, int KM, int NAM, int ROWS, int LMAX, int GMINB, bool FAST>
void launch_gather_tf(Engine& e, int N, double* pe, double* force, double* virial,
                      bool accumulate, cudaStream_t s)
{
  NeighborBuffers& nb = e.nbr;
  const int threads = 256;
  const int blocks = static_cast<int>((static_cast<long long>(N) * G + threads - 1) / threads);
  const int tt = e.params.T * e.params.T;
  const size_t smem =
    sizeof(float) * (2 * tt + 18 + (2 * tt + 18) % 4 +
                     (ROWS == kImages ? angular_table_floats(e.params, (KM + 3) & ~3) : 0));
  allow_smem(k_gather<G, KM, NAM, ROWS, LMAX, GMINB, FAST>, smem);
  k_gather<G, KM, NAM, ROWS, LMAX, GMINB, FAST><<<blocks, threads, smem, s>>>(
    e.params, N, e.d_box, e.scratch.sites, nb.nn_r, nb.nl_r, nb.mn_r, nb.nn_a, nb.nl_a, nb.mn_a,
    nb.st_a, nb.heads, nb.st_h, e.xr.er, e.xr.ea, e.scratch.acoef, e.scratch.alpha, e.scratch.f12, e.xr.large,
    e.scratch.pe_ann, pe,
    force, virial, accumulate ? 1 : 0, e.d_nstate);
}

template <int G, int KM, int NAM, int ROWS, int LMAX, int GMINB = 0>
void launch_gather_t(Engine& e, int N, double* pe, double* force, double* virial,
                     bool accumulate, cudaStream_t s)
{
  if constexpr (KM == kSmallK && LMAX == 4) {
    if (fast_math(e)) {
      // the FAST builds are held to their occupancy: two CTAs per SM on
      // rows of images, three for the uncapped Verlet-row build (it takes 84
      // registers unheld, which the 8-register allocation unit rounds to 88:
      // two CTAs of 256, and 1.5x the time)
      constexpr int fast_minb = ROWS == kImages ? 2 : (GMINB == 0 ? 3 : GMINB);
      launch_gather_tf<G, KM, NAM, ROWS, LMAX, fast_minb, true>(e, N, pe, force, virial,
                                                                accumulate, s);
      return;
    }
  }
  launch_gather_tf<G, KM, NAM, ROWS, LMAX, GMINB, false>(e, N, pe, force, virial, accumulate, s);
}

// the FP32 build or, for the mixed precisions, the tensor-core one
template <int G, int NRM, int KM, int NAM, int LMAX, int MINB>
void launch_fused_g(Engine& e, int N, cudaStream_t s)
{
  const bool tc = e.precision != 0;
  if (e.use_xr) {
    if (tc) launch_fused_t<G, NRM, KM, NAM, true, LMAX, MINB, true>(e, N, s);
    else launch_fused_t<G, NRM, KM, NAM, true, LMAX, MINB, false>(e, N, s);
  } else {
    if (tc) launch_fused_t<G, NRM, KM, NAM, false, LMAX, MINB, true>(e, N, s);
    else launch_fused_t<G, NRM, KM, NAM, false, LMAX, MINB, false>(e, N, s);
  }
}

// the general shape at 2 CTAs per SM (five n per moment sweep) or, with
// Engine::fused_minb 4, at 3 (three n): FP32; the tensor-core build comes at 2
// (13,824 carbon atoms at n_max 12 8, basis 16 12: 238 registers and 208 us of
// descriptor stage against 164 and 201; with the angular force inside 187)
template <int G>
void launch_fused_general(Engine& e, int N, cudaStream_t s)
{
  constexpr int n = kMaxN, k = kMaxBasis;
  if (!e.use_xr && e.fuse_f12) {
    if (e.precision != 0) launch_fused_t<G, n, k, n, false, 4, 2, true, true>(e, N, s);
    else if (e.fused_minb == 4) launch_fused_t<G, n, k, n, false, 4, 3, false, true>(e, N, s);
    else launch_fused_t<G, n, k, n, false, 4, 2, false, true>(e, N, s);
    return;
  }
  if (e.fused_minb == 4 && e.precision == 0) {
    if (e.use_xr) launch_fused_t<G, n, k, n, true, 4, 3, false>(e, N, s);
    else launch_fused_t<G, n, k, n, false, 4, 3, false>(e, N, s);
  } else {
    launch_fused_g<G, n, k, n, 4, 2>(e, N, s);
  }
}

// the small shape at 3 or 4 CTAs per SM (Engine::fused_minb, autotuned; the
// tensor-core build comes at 3)
template <int G>
void launch_fused_small(Engine& e, int N, cudaStream_t s)
{
  if (!e.use_xr && e.fuse_f12) {
    constexpr int n = kSmallN, k = kSmallK;
    if (e.precision != 0) launch_fused_t<G, n, k, n, false, 4, 3, true, true>(e, N, s);
    else if (e.fused_minb == 4) launch_fused_t<G, n, k, n, false, 4, 4, false, true>(e, N, s);
    else launch_fused_t<G, n, k, n, false, 4, 3, false, true>(e, N, s);
    return;
  }
  if (e.fused_minb == 4 && e.precision == 0) {
    if (e.use_xr) launch_fused_t<G, kSmallN, kSmallK, kSmallN, true, 4, 4, false>(e, N, s);
    else launch_fused_t<G, kSmallN, kSmallK, kSmallN, false, 4, 4, false>(e, N, s);
  } else {
    launch_fused_g<G, kSmallN, kSmallK, kSmallN, 4, 3>(e, N, s);
  }
}

// groups of 16 and 32: three CTAs per SM, the angular force inside on Verlet rows
template <int G>
void launch_fused_wide(Engine& e, int N, cudaStream_t s)
{
  constexpr int n = kSmallN, k = kSmallK;
  if (e.use_xr) launch_fused_tx<G, n, k, n, true, 4, 3, false, false, true>(e, N, s);
  else if (e.fuse_f12) launch_fused_tx<G, n, k, n, false, 4, 3, false, true, true>(e, N, s);
  else launch_fused_tx<G, n, k, n, false, 4, 3, false, false, true>(e, N, s);
}

template <int G, int KM, int NAM, int LMAX>
void launch_gather_xr(Engine& e, int N, double* pe, double* force, double* virial,
                      bool accumulate, cudaStream_t s)
{
  // a single system takes the images' scheme whatever its box
  if (e.xr.from_box || (e.xr.kinds & kSmallRows))
    launch_gather_t<G, KM, NAM, kImages, LMAX, 0>(e, N, pe, force, virial, accumulate, s);
  if (e.xr.from_box || !(e.xr.kinds & kLargeRows)) return;
  launch_gather_t<G, KM, NAM, kLarge, LMAX, LMAX == 4 ? 4 : 0>(e, N, pe, force, virial, accumulate,
                                                                s);
}

template <int G, int KM, int NAM, int LMAX>
void launch_gather_g(Engine& e, int N, double* pe, double* force, double* virial,
                     bool accumulate, cudaStream_t s)
{
  if (e.use_xr) {
    launch_gather_xr<G, KM, NAM, LMAX>(e, N, pe, force, virial, accumulate, s);
    return;
  }
  if constexpr (LMAX == 4) {
    if (e.gather_minb == 4) {
      launch_gather_t<G, KM, NAM, kVerlet, LMAX, 4>(e, N, pe, force, virial, accumulate, s);
      return;
    }
  }
  launch_gather_t<G, KM, NAM, kVerlet, LMAX, 0>(e, N, pe, force, virial, accumulate, s);
}

}  // namespace

#include "invariants_upload.inc"

// Padded basis width (row stride of the coefficient tables and of alpha).
int basis_stride(const ModelParams& p) { return small_shape(p) ? round4(kSmallK) : round4(kMaxBasis); }

int alpha_stride(const ModelParams& p)
{
  return small_shape(p) ? alpha_row<kSmallK>() : alpha_row<kMaxBasis>();
}

bool fused_occupancy_variants(const ModelParams& p) { return !high_degree(p); }

bool wide_groups(const ModelParams& p) { return small_shape(p); }

bool fused_wide_groups(const Engine& e) { return exact_shape(e.params) && e.precision == 0; }

// Largest dynamic shared memory a descriptor-kernel variant this model runs needs.
size_t fused_smem_bytes(const ModelParams& p)
{
  if (high_degree(p))
    return fused_layout(p, kBlock / kHighFusedGroup, basis_stride(p), fused_smem_budget(2), false)
      .total_bytes;
  return fused_layout(p, kBlock / 4, basis_stride(p), fused_smem_budget(small_shape(p) ? 3 : 2),
                      false)
    .total_bytes;
}

void set_fused_smem_limits(const ModelParams& p)
{
  // the tensor-core builds' layout needs the 16-bit tile sizes of the current
  // precision (set before this is called again by nepx_set_precision)
  const bool tc = p.tc_dimk > 0;
  if (high_degree(p)) {
    set_fused_smem_t<kHighFusedGroup, kMaxN, kMaxBasis, kMaxN, 8, 2, false>(p);
    if (tc) set_fused_smem_t<kHighFusedGroup, kMaxN, kMaxBasis, kMaxN, 8, 2, true>(p);
    return;
  }
  if (small_shape(p)) {
    set_fused_smem_wide<16>(p);
    set_fused_smem_wide<32>(p);
    set_fused_smem_t<4, kSmallN, kSmallK, kSmallN, 4, 3, false, true>(p);
    set_fused_smem_t<8, kSmallN, kSmallK, kSmallN, 4, 3, false, true>(p);
    set_fused_smem_t<4, kSmallN, kSmallK, kSmallN, 4, 4, false, true>(p);
    set_fused_smem_t<8, kSmallN, kSmallK, kSmallN, 4, 4, false, true>(p);
    if (tc) {
      set_fused_smem_t<4, kSmallN, kSmallK, kSmallN, 4, 3, true, true>(p);
      set_fused_smem_t<8, kSmallN, kSmallK, kSmallN, 4, 3, true, true>(p);
    }
  } else {
    set_fused_smem_t<4, kMaxN, kMaxBasis, kMaxN, 4, 2, false, true>(p);
    set_fused_smem_t<8, kMaxN, kMaxBasis, kMaxN, 4, 2, false, true>(p);
    set_fused_smem_t<4, kMaxN, kMaxBasis, kMaxN, 4, 3, false, true>(p);
    set_fused_smem_t<8, kMaxN, kMaxBasis, kMaxN, 4, 3, false, true>(p);
    if (tc) {
      set_fused_smem_t<4, kMaxN, kMaxBasis, kMaxN, 4, 2, true, true>(p);
      set_fused_smem_t<8, kMaxN, kMaxBasis, kMaxN, 4, 2, true, true>(p);
    }
  }
}

size_t fused_tc_smem_bytes(const ModelParams& p)
{
  if (high_degree(p))
    return fused_layout(p, kBlock / kHighFusedGroup, basis_stride(p), fused_smem_budget(2), true)
      .total_bytes;
  return fused_layout(p, kBlock / 4, basis_stride(p), fused_smem_budget(small_shape(p) ? 3 : 2),
                      true)
    .total_bytes;
}

void launch_filter(Engine& e, int N, cudaStream_t s)
{
  const bool small = small_shape(e.params);
  if (small && e.filter_group == 32) launch_filter_t<32, kSmallN, kSmallK>(e, N, s);
  else if (small && e.filter_group == 16) launch_filter_t<16, kSmallN, kSmallK>(e, N, s);
  else if (e.filter_group >= 8) {
    if (small) launch_filter_t<8, kSmallN, kSmallK>(e, N, s);
    else launch_filter_t<8, kMaxN, kMaxBasis>(e, N, s);
  } else {
    if (small) launch_filter_t<4, kSmallN, kSmallK>(e, N, s);
    else launch_filter_t<4, kMaxN, kMaxBasis>(e, N, s);
  }
}

// The descriptor kernel evaluates the angular partial forces itself (degrees
// <= 4, Verlet rows, when the autotuner picked it).
bool fused_angular_force(const Engine& e)
{
  return e.fuse_f12 && !e.use_xr && !high_degree(e.params);
}

void launch_descriptor(Engine& e, int N, const double*, const int*, cudaStream_t stream)
{
  const bool small = small_shape(e.params);
  const bool high = high_degree(e.params);
  if (!e.use_xr) {
    launch_filter(e, N, stream);
    if (e.nbr.heads_after_filter) {
      const NeighborBuffers& nb = e.nbr;
      const long long slots = static_cast<long long>(N) * (1 + nb.st_a / 8);
      k_row_heads<<<static_cast<unsigned>((slots + 255) / 256), 256, 0, stream>>>(
        N, nb.nn_a, nb.nl_a, nb.st_a, nb.heads, nb.st_h);
    }
  }
  if (high) launch_fused_g<kHighFusedGroup, kMaxN, kMaxBasis, kMaxN, 8, 2>(e, N, stream);
  else if (e.group == 32 && fused_wide_groups(e)) launch_fused_wide<32>(e, N, stream);
  else if (e.group == 16 && fused_wide_groups(e)) launch_fused_wide<16>(e, N, stream);
  else if (e.group >= 8) {
    if (small) launch_fused_small<8>(e, N, stream);
    else launch_fused_general<8>(e, N, stream);
  } else {
    if (small) launch_fused_small<4>(e, N, stream);
    else launch_fused_general<4>(e, N, stream);
  }
  // a single explicit-row system: the gather evaluates both directed angular
  // forces itself; a batch's structures that are not small take f12 here
  if (e.use_xr && (e.xr.from_box || !(e.xr.kinds & kLargeRows))) return;
  if (fused_angular_force(e)) return;   // the descriptor kernel wrote f12
  if (high) launch_f12_t<kHighGroup, kMaxBasis, kMaxN, 8>(e, N, stream);
  else if (e.f12_group >= 8) {
    if (small) launch_f12_t<8, kSmallK, kSmallN, 4>(e, N, stream);
    else launch_f12_t<8, kMaxBasis, kMaxN, 4>(e, N, stream);
  } else {
    if (small) launch_f12_t<4, kSmallK, kSmallN, 4>(e, N, stream);
    else launch_f12_t<4, kMaxBasis, kMaxN, 4>(e, N, stream);
  }
}

void launch_gather(Engine& e, int N, const double*, const int*, double* pe, double* force,
                   double* virial, bool accumulate, cudaStream_t stream)
{
  const bool small = small_shape(e.params);
  if (high_degree(e.params))
    launch_gather_g<kHighGroup, kMaxBasis, kMaxN, 8>(e, N, pe, force, virial, accumulate, stream);
  else if (small && e.gather_group == 32)
    launch_gather_g<32, kSmallK, kSmallN, 4>(e, N, pe, force, virial, accumulate, stream);
  else if (small && e.gather_group == 16 && e.use_xr)   // (no choice takes 16 on Verlet rows)
    launch_gather_xr<16, kSmallK, kSmallN, 4>(e, N, pe, force, virial, accumulate, stream);
  else if (e.gather_group == 4) {
    if (small) launch_gather_g<4, kSmallK, kSmallN, 4>(e, N, pe, force, virial, accumulate, stream);
    else launch_gather_g<4, kMaxBasis, kMaxN, 4>(e, N, pe, force, virial, accumulate, stream);
  } else {
    if (small) launch_gather_g<8, kSmallK, kSmallN, 4>(e, N, pe, force, virial, accumulate, stream);
    else launch_gather_g<8, kMaxBasis, kMaxN, 4>(e, N, pe, force, virial, accumulate, stream);
  }
}

void launch_force(Engine& e, int N, const double* pos, const int* type, double* pe,
                  double* force, double* virial, bool accumulate, cudaStream_t stream)
{
  launch_descriptor(e, N, pos, type, stream);
  launch_gather(e, N, pos, type, pe, force, virial, accumulate, stream);
}

}  // namespace nepx
