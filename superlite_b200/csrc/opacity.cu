// opacity.cu -- physical LTE opacity (bound-bound expansion opacity binned into
// groups, Verner bound-free, Sutherland free-free), analytic opacity and the
// Planck / Rosseland means, for sm_100a.
//
// Reference: GAS/physical_opacity.f:3-357, bfxsmod.f:65-153,
// GAS/analytic_opacity.f90:3-77, GAS/opacity_planckmean.f:17-24,
// GAS/opacity_rossmean.f:17-21.
//
// Design (one B200):
//  * What depends on the line list, the bound-free fits and the group grid alone
//    is laid out once after slg_set_groups / slg_set_atomic_data (opacity_plan):
//    the sub-groups' line ranges, each line's 16-byte record with its
//    sub-group's lines ordered by the population row they multiply, and the
//    cross sections of every sub-group and ion.
//  * opac_cell: the shells' scalars, populations and free-free sums; bf_select: the
//    populated ions' nonzero cross sections of every sub-group.
//  * opacity_fwd: one warp per (group, 32 FS shells).  Every lane walks the
//    lines of its group (warp-uniform broadcast reads) and accumulates bb row
//    by row, then bf (ions in the reference's iz,ii order), then ff (elements
//    summed per shell beforehand) into one register per shell.  Sub-groups are
//    collapsed in registers.  A shell's values go to memory one by one: its
//    neighbouring groups are the neighbouring blocks', and the parts of a sector
//    meet in L2.
//  * FP64 throughout, compiled without FMA contraction; the bb and bf sums use
//    explicit fused multiply-adds and bb sums run row by row, so opacities agree
//    with the single-threaded Fortran to rounding (1e-12 relative is tested), not
//    to the bit.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <algorithm>
#include <cfloat>
#include "slg_device.cuh"
#include "slg_internal.h"

namespace slg {

namespace {

// Builds with lines take up to this many sub-groups and refuse more.  Nothing here
// needs the limit (an earlier layout held the edges in shared memory); callers see the
// same sizes accepted and refused as ever.
constexpr int kMaxLineSubgroups = 18770;
constexpr int OPAC_CT = 32;  // lanes of a warp, each with one or more shells

// ------------------------------------------------------------ line ranges
// lstart[igs] (igs = 0..nedge+1) = first line whose sub-group pointer
// (physical_opacity.f:117-125: igs = #{k : wlsub(k) <= wl0}) is at least igs;
// the lines are sorted by wl0 (slg_set_atomic_data), so it is the first line
// at or above edge igs-1.
__global__ void line_range_kernel(const slg_bbxs* __restrict__ bb, int64_t nline, const double* __restrict__ wlsub,
                                  int nedge, int* __restrict__ lstart) {
  const int igs = blockIdx.x * blockDim.x + threadIdx.x;
  if (igs > nedge + 1) return;
  int64_t lo = 0, hi = igs == 0 ? 0 : nline;
  if (igs > nedge) lo = nline;
  const double edge = igs >= 1 && igs <= nedge ? wlsub[igs - 1] : 0.0;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((double)bb[mid].wl0 * pc_ang >= edge) hi = mid;
    else lo = mid + 1;
  }
  lstart[igs] = (int)lo;
}

// ------------------------------------------------------------ per-cell preparation
// hckt (physical_opacity.f:81), gas_sig (:84-89), hlparr (:203), grndlev (:95-101,
// :165-171), which ion slots (iz,ii) carry any population (active, zeroed by the
// caller), and per (cell, element) the free-free Gaunt columns (:226-231).
//
// Free-free, summed over elements once per shell.  For fixed table columns
// (igg, dgg) of each element, the reference's bilinear gff (physical_opacity.f:
// 234-237) is linear in the row weights (1 - du, du):
//   g_z = (1 - du) Gz[iu - 1] + du Gz[iu],  Gz[j] = (1 - dgg) G[j, igg - 1] + dgg G[j, igg],
// so sum_z z^2 fr_z g_z = (1 - du) S[iu - 1] + du S[iu] with
// S[j] = sum_z z^2 fr_z Gz[j] over the elements without the gff >= 1 clamp
// (:238, nonlinear); those are flagged in ffclamp (bit iz - 1) and added per
// group.  Elements with fr = 0 add +0 in the reference (:240-241) and are left
// out.  The sum is re-associated (one product by help per group instead of one
// per element): a rounding-level difference.  For the adjoint: D[j] = sum_z
// z^2 fr_z (G[j, igg] - G[j, igg - 1]) over the same elements (d gff / d dgg
// is linear in the row weights too), and ffclamp_all flags every clamped
// element whatever its fr (d cap / d fr needs them all).
//
// A block takes CELLS shells: first the populations, shells fastest, then a warp
// per shell: a lane per element finds its columns, the elements that enter the
// sums are compacted into shared memory, and the lanes take the 81 table rows.
// (Cold caches, under the profiler: as one thread per (shell, row) that walked all
// elements the sums alone took 17-20 us whatever the grid, besides 9 us for the rest;
// now 12 us in all at 256 shells, 18 at 4096.)
constexpr int CELLS = 8;
// Length of a population row: whole warps' shells (64 of two per lane, 32 up to 32
// shells, which are one per lane).
static int padded_shells(int nc) { return nc <= OPAC_CT ? OPAC_CT : (nc + 2 * OPAC_CT - 1) / (2 * OPAC_CT) * (2 * OPAC_CT); }
__global__ void __launch_bounds__(CELLS * 32) opac_cell_kernel(
    int nc, int nelem, int nst, const int32_t* __restrict__ ion_ni, const double* __restrict__ temp,
    const double* __restrict__ natom, const double* __restrict__ nelec, const double* __restrict__ vol,
    const double* __restrict__ mass, const double* __restrict__ oc, const double* __restrict__ ginv, int nothmson,
    const double* __restrict__ natomfr, const double* __restrict__ G, double* __restrict__ hckt,
    double* __restrict__ gas_sig, double* __restrict__ hlparr, int ld, int nrow,
    const int16_t* __restrict__ slot_of_row, double* __restrict__ grndlev,
    double* __restrict__ ocp, int* __restrict__ active, int* __restrict__ ffigg, double* __restrict__ ffdgg, double* __restrict__ ffsum,
    double* __restrict__ ffdsum, unsigned* __restrict__ ffclamp, unsigned* __restrict__ ffclamp_all) {
  __shared__ double s_w[CELLS][32], s_dgg[CELLS][32];
  __shared__ int s_igg[CELLS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nslot = nelem * nst;
  for (int t = threadIdx.x; t < nslot * CELLS; t += CELLS * 32) {  // a multiple of CELLS per slot
    const int k = t / CELLS, i = blockIdx.x * CELLS + t % CELLS;
    const double o = i < nc ? oc[(size_t)k * nc + i] : 0.0;
    if (i < ld) ocp[(size_t)k * ld + i] = o;
    if (o != 0.0) active[k] = 1;
  }
  for (int t = threadIdx.x; t < nrow * CELLS; t += CELLS * 32) {  // the lines' population rows
    const int row = t / CELLS, k = slot_of_row[row], i = blockIdx.x * CELLS + t % CELLS;
    double v = 0.0;
    if (i < nc) {
      const int iz = k / nst + 1, ii = k % nst + 1;
      if (ii <= min(iz, ion_ni[iz - 1] - 1) && mass[i] > 0.0) v = oc[(size_t)k * nc + i] * ginv[(size_t)k * nc + i];
    }
    if (i < ld) grndlev[(size_t)row * ld + i] = v < 0.0 ? 0.0 : v;  // the reference skips lines with ocg <= 0
  }
  const int i = blockIdx.x * CELLS + warp;
  if (i >= nc) return;  // uniform over the warp
  const double h = pc_hc / (pc_kb * temp[i]);
  if (lane == 0) {
    hckt[i] = h;
    double s = 0.0;
    if (!nothmson) {
      s = cthomson * nelec[i] * natom[i] / vol[i];
      if (mass[i] <= 0.0) s = 0.0;
    }
    gas_sig[i] = s;
    hlparr[i] = sq(natom[i] / vol[i]) * nelec[i];
  }
  if (!G) return;
  bool clamped = false, in_sum = false;
  double fr = 0.0, dgg = 0.0;
  int igg = 1;
  if (lane < nelem) {
    const int iz = lane + 1;
    const double gg = (double)(iz * iz) * pc_rydberg * h;
    const double rgg = 5.0 * (log10(gg) + 4.0) + 1.0;
    // max(floor(rgg), 1) and min(., ff_ngg - 1) as :228-230; a NaN (from a NaN
    // temperature) takes the lower bound, so the table reads stay in bounds
    igg = !(rgg >= 1.0) ? 1 : (rgg >= (double)(FF_NGG - 1) ? FF_NGG - 1 : (int)floor(rgg));
    dgg = rgg - igg;
    clamped = rgg > (double)FF_NGG;
    ffigg[(size_t)lane * nc + i] = clamped ? -igg : igg;  // sign: gff >= 1 clamp (:238)
    ffdgg[(size_t)lane * nc + i] = dgg;
    fr = natomfr[(size_t)(nelem + 1) * i + iz];
    in_sum = fr != 0.0 && !clamped;
  }
  const unsigned m_sum = __ballot_sync(0xffffffffu, in_sum);
  const unsigned m_all = __ballot_sync(0xffffffffu, clamped), m_fr = __ballot_sync(0xffffffffu, clamped && fr != 0.0);
  if (in_sum) {
    const int q = __popc(m_sum & ((1u << lane) - 1u));
    s_w[warp][q] = (double)((lane + 1) * (lane + 1)) * fr;
    s_dgg[warp][q] = dgg;
    s_igg[warp][q] = igg;
  }
  __syncwarp();
  const int n = __popc(m_sum);
  for (int j = lane; j < FF_NU; j += 32) {
    double S = 0.0, D = 0.0;
#pragma unroll 4
    for (int q = 0; q < n; ++q) {
      const double* g = G + j + FF_NU * (s_igg[warp][q] - 1);
      const double g0 = g[0], g1 = g[FF_NU], d = s_dgg[warp][q], w = s_w[warp][q];
      const double gz = (1.0 - d) * g0 + d * g1;
      S = S + w * gz;
      D = D + w * (g1 - g0);
    }
    ffsum[(size_t)i * FF_NU + j] = S;
    ffdsum[(size_t)i * FF_NU + j] = D;
  }
  if (lane == 0) {
    ffclamp[i] = m_fr;
    ffclamp_all[i] = m_all;
  }
}

// Active slots in the reference's loop order (iz ascending, ii = 1..min(iz,ni-1)),
// physical_opacity.f:180-181: that order is increasing slot = (iz-1) nst + (ii-1),
// so one warp compacts the valid, populated slots 32 at a time with a ballot.
__global__ void ion_compact_kernel(int nelem, int nst, const int32_t* __restrict__ ion_ni,
                                   const int* __restrict__ active, int16_t* __restrict__ act_slot,
                                   int* __restrict__ nact) {
  const int lane = threadIdx.x & 31;
  const int nslot = nelem * nst;
  int n = 0;
  for (int k0 = 0; k0 < nslot; k0 += 32) {
    const int k = k0 + lane;
    bool ok = false;
    if (k < nslot) {
      const int iz = k / nst + 1, ii = k % nst + 1;
      ok = ii <= min(iz, ion_ni[iz - 1] - 1) && active[k] != 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (ok) act_slot[n + __popc(m & ((1u << lane) - 1u))] = (int16_t)k;
    n += __popc(m);
  }
  if (lane == 0) *nact = n;
}

// Sub-group edges wlsub (physical_opacity.f:65-78), padded with DBL_MAX.
__global__ void wlsub_kernel(int ng, int ngs, int nedge_pad, const double* __restrict__ wl,
                             double* __restrict__ wlsub) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;  // 0-based edge
  if (k >= nedge_pad) return;
  const int nedge = ng * ngs + 1;
  double v = DBL_MAX;
  if (k < nedge) {
    if (ngs == 1 || k == 0) {
      v = wl[ngs == 1 ? k : 0];
    } else {
      const int ig = (k - 1) / ngs + 1, i = (k - 1) % ngs + 1;
      const double help = 1.0 / ngs;
      v = (1.0 - i * help) * wl[ig - 1] + i * help * wl[ig];
    }
  }
  wlsub[k] = v;
}

// ------------------------------------------------------------ bound-free cross sections
__device__ inline float PH1(const float* t, int k, int is, int nz, int ne) {
  return t[(k - 1) + 6 * ((is - 1) + 7 * ((nz - 1) + 30 * (ne - 1)))];
}
__device__ inline float PH2(const float* t, int k, int nz, int ne) {
  return t[(k - 1) + 7 * ((nz - 1) + 30 * (ne - 1))];
}
__device__ inline float sqf(float x) { return __fmul_rn(x, x); }  // real*4 ** 2

// bfxsmod.f:65-153
__device__ double bfxs(const float* __restrict__ ph1, const float* __restrict__ ph2, int nz, int ne,
                       double e) {
  const int ll[7] = {0, 0, 1, 0, 1, 2, 0};
  const int ninn[30] = {0, 0, 1, 1, 1, 1, 1, 1, 1, 1, 3, 3, 3, 3, 3,
                        3, 3, 3, 5, 5, 5, 5, 5, 5, 5, 5, 5, 5, 5, 5};
  const int ntot[30] = {1, 1, 2, 2, 3, 3, 3, 3, 3, 3, 4, 4, 5, 5, 5,
                        5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 6, 6, 6, 7, 7};
  double xs = 0.0;
  if (nz < 1 || nz > 30) return xs;
  if (ne < 1 || ne > nz) return xs;
  int nout = ntot[ne - 1];
  if (nz > 18) {
    if (nz == ne) nout = 7;
    if (nz == ne + 1 && (nz == 20 || nz == 21 || nz == 22 || nz == 25 || nz == 26)) nout = 7;
  }
  if (e < (double)PH1(ph1, 1, nout, nz, ne)) return xs;
  const int nint_ = ninn[ne - 1];
  double einn;
  if (nz == 15 || nz == 17 || nz == 19 || (nz > 20 && nz != 26)) einn = 0.0;
  else einn = ne < 3 ? (double)1.0e30f : (double)PH1(ph1, 1, nint_, nz, ne);
  for (int is = 1; is <= nout; ++is) {
    if (e < (double)PH1(ph1, 1, is, nz, ne)) continue;
    if (is < nout && is > nint_ && e < einn) continue;
    if (is <= nint_ || e >= einn) {
      const double p1 = -(double)PH1(ph1, 5, is, nz, ne);
      const double y = e / (double)PH1(ph1, 2, is, nz, ne);
      const double q = -0.5 * p1 - (double)ll[is - 1] - 5.5;
      const double a = (double)PH1(ph1, 3, is, nz, ne) * (sq(y - 1.0) + (double)sqf(PH1(ph1, 6, is, nz, ne)));
      const double b = sqrt(y / (double)PH1(ph1, 4, is, nz, ne)) + 1.0;
      xs = xs + a * pow(y, q) * pow(b, p1);
    } else {
      const double p1 = -(double)PH2(ph2, 4, nz, ne);
      const double q = -0.5 * p1 - 5.5;
      const double x = e / (double)PH2(ph2, 1, nz, ne) - (double)PH2(ph2, 6, nz, ne);
      const double z = sqrt(x * x + (double)sqf(PH2(ph2, 7, nz, ne)));
      const double a = (double)PH2(ph2, 2, nz, ne) * (sq(x - 1.0) + (double)sqf(PH2(ph2, 5, nz, ne)));
      const double b = 1.0 + sqrt(z / (double)PH2(ph2, 3, nz, ne));
      xs = xs + a * pow(z, q) * pow(b, p1);
    }
  }
  return xs;
}

// xstab[(igs-1) nslot + slot] = bfxs(iz, iz-ii+1, hc/(ev*wlsub(igs))) * pc_mbarn,
// :177-186 (the reference's first product), for every slot that the reference
// visits (ii <= min(iz, ni-1)), else 0.  Without the fits (slg_set_atomic_data took
// null) a cross section is not a number: a build whose ions have no population needs
// none, any other gets NaN, which its sanity word reports.
__global__ void bf_table_kernel(int ngsub, int nslot, const int32_t* __restrict__ ion_ni, int nst,
                                const double* __restrict__ wlsub, const float* __restrict__ ph1,
                                const float* __restrict__ ph2, double* __restrict__ xstab) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)ngsub * nslot) return;
  const int igs = (int)(t / nslot) + 1;
  const int slot = (int)(t % nslot);
  const int iz = slot / nst + 1, ii = slot % nst + 1;
  double x = 0.0;
  if (ii <= min(iz, ion_ni[iz - 1] - 1))
    x = ph1 && ph2 ? bfxs(ph1, ph2, iz, iz - ii + 1, pc_hc / (pc_ev * wlsub[igs - 1])) * pc_mbarn : CUDART_NAN;
  xstab[t] = x;
}

// One nonzero bound-free cross section of a sub-group (times pc_mbarn) and the
// ion slot whose population it multiplies: one vector load.
struct __align__(16) BfTerm {
  double xs;
  int slot, pad;
};

// Per sub-group, its nonzero cross sections whose ion carries any population, in
// slot order (the reference's loop order; it skips xs == 0,
// physical_opacity.f:184, and a term of an unpopulated ion adds +0), one warp
// per sub-group.
__global__ void bf_select_kernel(int ngsub, int nslot, int maxbf, const double* __restrict__ xstab,
                                 const int* __restrict__ active, BfTerm* __restrict__ terms,
                                 int* __restrict__ count) {
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= ngsub) return;
  const size_t base = (size_t)w * nslot, out = (size_t)w * maxbf;
  int k = 0;
  for (int a0 = 0; a0 < nslot; a0 += 32) {
    const int a = a0 + lane;
    const double x = a < nslot ? xstab[base + a] : 0.0;
    const bool on = x != 0.0 && active[a] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) terms[out + k + __popc(m & ((1u << lane) - 1u))] = BfTerm{x, a, 0};
    k += __popc(m);
  }
  if (lane == 0) count[w] = k;
}

// One line's shell-independent factors, 16 bytes (one vector load per line):
// pg = phi(igs) * gxs, the first product of the reference's expression
// (physical_opacity.f:148-149), so the evaluation order of that product is
// kept, times kPgScale; and chilw in FP64 with two indices in the low 29 bits of its
// mantissa.  chilw is single precision in the line record (as in the
// reference's bbxs type), so those bits of its FP64 value are zero: masking
// them off gives chilw exactly, without a conversion per line.  The indices:
// bits 0..10 the line's row among the population rows the lines reference
// (lrow_of_slot), bits 11..26 its population slot (iz - 1) nst + (ii - 1), bit
// 27 set on the last line of its row in its sub-group: a sub-group's lines are
// ordered by row, so that a sum over lines takes each population once per row.
struct __align__(16) LineTerm {
  double pg;
  double chi_idx;
};
// Keeps pg exp(-chi h) a normal number for the smallest exp (1e-304; pg alone is about
// 1e-12, and the population comes after the sum over a row); a power of two, so that
// nothing rounds otherwise.  Taken off the sums by kPgUnscale.
constexpr double kPgScale = 0x1p100, kPgUnscale = 0x1p-100;
constexpr int kLineRowBits = 11;
constexpr unsigned kLineIdxMask = 0x1fffffffu;
constexpr unsigned kLineRowEnd = 1u << 27;

struct LineVals {
  double pg, chi;
  unsigned idx;
};

__device__ __forceinline__ LineVals load_line(const LineTerm* p) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(p));
  const unsigned lo = (unsigned)__double2loint(v.y);
  return LineVals{v.x, __hiloint2double(__double2hiint(v.y), (int)(lo & ~kLineIdxMask)), lo & kLineIdxMask};
}
__device__ __forceinline__ int line_slot(unsigned idx) { return (int)((idx >> kLineRowBits) & 0xffffu); }
__device__ __forceinline__ int line_row(unsigned idx) { return (int)(idx & ((1u << kLineRowBits) - 1u)); }

// The LineTerms of sub-group w + 1, one warp each: its lines counted by row,
// the rows' first places, then the lines written there in file order (a lane's
// place within a round of 32 is its rank among the lanes of the same row), so
// the layout does not depend on timing.  Dynamic shared memory: nrow ints per warp.
constexpr int LT_WARPS = 4;
__global__ void __launch_bounds__(LT_WARPS * 32) line_terms_kernel(const slg_bbxs* __restrict__ bb,
                                                                   const int* __restrict__ lstart,
                                                                   int ngsub,
                                                                   const double* __restrict__ wlsub, int nst,
                                                                   const int16_t* __restrict__ lrow_of_slot, int nrow,
                                                                   LineTerm* __restrict__ lt) {
  extern __shared__ int s_at[];
  const int w = blockIdx.x * LT_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  int* at = s_at + (size_t)(threadIdx.x >> 5) * nrow;
  if (w >= ngsub) return;
  const int igs = w + 1, l0 = lstart[igs], l1 = lstart[igs + 1];
  for (int r = lane; r < nrow; r += 32) at[r] = 0;
  __syncwarp();
  for (int l = l0 + lane; l < l1; l += 32) atomicAdd(&at[lrow_of_slot[(bb[l].iz - 1) * nst + (bb[l].ii - 1)]], 1);
  __syncwarp();
  int sum = l0;
  for (int r0 = 0; r0 < nrow; r0 += 32) {  // exclusive scan of the counts
    const int n = r0 + lane < nrow ? at[r0 + lane] : 0;
    int inc = n;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (r0 + lane < nrow) at[r0 + lane] = sum + inc - n;
    sum += __shfl_sync(0xffffffffu, inc, 31);
  }
  __syncwarp();
  const double wa = wlsub[igs - 1], wb = wlsub[igs];
  const double wl = 0.5 * (wa + wb);
  const double phi = wl * wl / ((wb - wa) * pc_c);
  for (int c0 = l0; c0 < l1; c0 += 32) {
    const int l = c0 + lane;
    slg_bbxs r{0.f, 0.f, 0.f, 1, 1};
    if (l < l1) r = bb[l];
    const int slot = (r.iz - 1) * nst + (r.ii - 1);
    const int row = l < l1 ? lrow_of_slot[slot] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, row);
    if (l < l1) {
      const int pos = at[row] + __popc(same & ((1u << lane) - 1u));
      const double chi = (double)r.chilw;  // low 29 mantissa bits zero
      const unsigned idx = ((unsigned)slot << kLineRowBits) | (unsigned)row;
      lt[pos] = LineTerm{phi * (double)r.gxs * kPgScale,
                         __hiloint2double(__double2hiint(chi), (int)((unsigned)__double2loint(chi) | idx))};
    }
    __syncwarp();
    if (l < l1 && (same & ((1u << lane) - 1u)) == 0u) at[row] += __popc(same);
    __syncwarp();
  }
  // at[r] is now the end of row r: mark the last line of each row
  __threadfence_block();
  __syncwarp();
  for (int r = lane; r < nrow; r += 32) {
    const int end = at[r], beg = r == 0 ? l0 : at[r - 1];
    if (end > beg) {
      const double x = lt[end - 1].chi_idx;
      lt[end - 1].chi_idx = __hiloint2double(__double2hiint(x), (int)((unsigned)__double2loint(x) | kLineRowEnd));
    }
  }
}

struct OpacArgs {
  int nc, ng, ngs, ngsub, nelem, nst, maxact;
  int maxbf;                // row length of bf: the slots that can have a cross section
  int nobb, nobf, noff;
  const int* pnact;         // number of active bound-free ion slots (device; adjoint)
  double mix;
  const double* wlsub;
  const double* grp_wl;
  const int* lstart;        // (ngsub+2)+1 line offsets by igs
  int ld;                   // row length of grndlev and ocp (padded_shells)
  const LineTerm* lt;       // per line, by sub-group and row (line_terms_kernel)
  double chimax;            // largest chilw of the lines (infinite: check every exp argument)
  const double* grndlev;    // [row of the lines' population rows][ld], negative values as zero
  const double* ocp;        // [slot][ld]
  const int* active;        // [slot]: nonzero if any cell has population there
  const int16_t* act_slot;  // the active slots, reference order (adjoint)
  const double* xstab;      // [(igs-1) nslot + slot]: bfxs * pc_mbarn
  const BfTerm* bf;         // [(igs-1) maxbf + k]: its nonzero entries of populated ions
  const int* bnnz;          // their count per sub-group
  const double* hckt;
  const double* hlparr;
  const double* mass;
  const double* natomfr;    // (0:nelem, ncell)
  const double* temp;
  const int* ffigg;         // [iz-1][cell], negative: apply gff >= 1
  const double* ffdgg;
  const double* ffsum;      // [cell][81]: sum over unclamped elements of z^2 fr gff at each table row
  const double* ffdsum;     // [cell][81]: the same of z^2 fr d gff / d dgg
  const unsigned* ffclamp;  // [cell]: elements (bit iz-1) with fr != 0 under the gff >= 1 clamp
  const unsigned* ffclamp_all;  // [cell]: every element under the clamp
  const double* gff;        // (81,41)
  double ffc1;
  float* cap32;             // (ng, ncell)
  float* emiss32;
  double* cap64;            // (ncell, ng) optional
  double* capg64 = nullptr; // (ng, ncell) optional: cap before sngl() in gas_cap's layout
  int* flags;
};

constexpr int kOpacWarps = 4;  // most warps of a forward or adjoint block
constexpr int kExpTabBytes = sizeof(double) * kExpTabN * kExpCopies;
// N neighbouring doubles, N * 8 bytes aligned (at most 16).
template <int N>
__device__ __forceinline__ void load_run(const double* __restrict__ p, double* v) {
  if (N == 1) {
    v[0] = __ldg(p);
  } else {
#pragma unroll
    for (int k = 0; k < N; k += 2) {
      const double2 d = __ldg(reinterpret_cast<const double2*>(p + k));
      v[k] = d.x;
      v[k + 1] = d.y;
    }
  }
}

// Bound-bound sums of a lane's FS neighbouring shells (pop: their first entry of
// the population rows, ld apart; arg: their exp arguments) over the n >= 1
// lines of a sub-group: per row sum of pg exp(-chi h), times the row's
// population, the rows added one after another by fused multiply-adds.  The
// next record and the next row's populations are loaded ahead.  (A loop per row:
// as a test after each line the row's end was compiled to predicated
// instructions that every line issued, 4 of 26 per term.)
template <int FS>
__device__ __forceinline__ void bb_sums(const LineTerm* __restrict__ lt, int n, const ExpArg* arg, const ExpConst& C,
                                        const double* __restrict__ pop, int ld, const double* s_tab, uint32_t mine,
                                        double* a) {
  double og[FS];
  LineVals t = load_line(lt);
  load_run<FS>(pop + (size_t)line_row(t.idx) * ld, og);
#pragma unroll
  for (int s = 0; s < FS; ++s) a[s] = 0.0;
  const LineTerm* const end = lt + n;
  do {
    double acc[FS];
#pragma unroll
    for (int s = 0; s < FS; ++s) acc[s] = 0.0;
#pragma unroll 1
    for (;;) {
      const LineVals u = load_line(lt + 1);
#pragma unroll
      for (int s = 0; s < FS; ++s) acc[s] = fma(t.pg, exp_scaled(t.chi, arg[s], C, s_tab, mine), acc[s]);
      ++lt;
      if (t.idx & kLineRowEnd) {  // the same for the whole warp
        t = u;
        break;
      }
      t = load_line(lt + 1);
#pragma unroll
      for (int s = 0; s < FS; ++s) acc[s] = fma(u.pg, exp_scaled(u.chi, arg[s], C, s_tab, mine), acc[s]);
      ++lt;
      if (u.idx & kLineRowEnd) break;
    }
#pragma unroll
    for (int s = 0; s < FS; ++s) a[s] = fma(acc[s], og[s], a[s]);
    load_run<FS>(pop + (size_t)line_row(t.idx) * ld, og);  // (any row's where none follows)
  } while (lt < end);
}
// The sum of one shell of a warp with one whose arguments may leave exp_scaled's
// range (or are not numbers): out of line and in few registers, so that the loop
// of all other warps keeps its own (inlined, or with two shells at once, it cost
// that loop 6 to 13 %), and to the same bits, so that a shell's value does not
// depend on the warp it is in.  256 shells x 2000 groups, a fourth of the shells beyond
// the range: 341 us a build, with exp for every term of such a warp 401.
__device__ __noinline__ double bb_sum_any(const LineTerm* __restrict__ lt, int n, double h,
                                          const double* __restrict__ pop, int ld) {
  extern __shared__ double etab[];  // opacity_fwd_kernel's
  double a = 0.0, acc = 0.0;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const LineVals t = load_line(lt + k);
    const double x = t.chi * h;
    double e;
    if (fabs(x) <= 700.0) e = exp_scaled(t.chi, exp_arg(h), ExpConst{}, etab, exp_table_mine());
    else e = x > 746.0 ? 0.0 : exp(-x);  // (exp's zero, without its call)
    acc = fma(t.pg, e, acc);
    if (t.idx & kLineRowEnd) {
      a = fma(acc, __ldg(pop + (size_t)line_row(t.idx) * ld), a);
      acc = 0.0;
    }
  }
  return a;
}
// Free-free of sub-group igs for shell i (h = hc/kT), added to cap.
__device__ inline double ff_add(const OpacArgs& A, int i, int igs, double h, double cap) {
  if (!A.noff) {
    const double wl = A.wlsub[igs - 1];
    const double wlinv = 1.0 / wl;
    const double u = h * wlinv;
    const double ru = 10.0 * (log10(u) + 4.0) + 1.0;
    const int iu = !(ru >= 1.0) ? 1 : (ru >= (double)(FF_NU - 1) ? FF_NU - 1 : (int)floor(ru));
    const double du = ru - iu;
    const double help = A.ffc1 * sqrt(h) * (1.0 - exp(-u)) * cube(wl) * A.hlparr[i];
    // sum over elements of z^2 fr gff (opac_cell_kernel), the clamped ones here
    const double* S = A.ffsum + (size_t)i * FF_NU;
    double sg = (1.0 - du) * __ldg(S + iu - 1) + du * __ldg(S + iu);
    for (unsigned m = __ldg(A.ffclamp + i); m; m &= m - 1) {
      const int iz = __ffs(m);
      const int igg = -A.ffigg[(size_t)(iz - 1) * A.nc + i];
      const double dgg = A.ffdgg[(size_t)(iz - 1) * A.nc + i];
      const double* G = A.gff;
      double g = (1.0 - du) * (1.0 - dgg) * G[(iu - 1) + FF_NU * (igg - 1)] +
                 du * (1.0 - dgg) * G[iu + FF_NU * (igg - 1)] +
                 (1.0 - du) * dgg * G[(iu - 1) + FF_NU * igg] + du * dgg * G[iu + FF_NU * igg];
      g = g > 1.0 ? g : 1.0;
      sg = sg + (double)(iz * iz) * A.natomfr[(size_t)(A.nelem + 1) * i + iz] * g;
    }
    cap = cap + help * sg;
  }
  return cap;
}

// 1 - exp(-h / wl(igs)), wl the sub-group's centre: the stimulated-emission
// factor of the bound-bound term (physical_opacity.f:148-149).
__device__ __forceinline__ double bb_expfac(const OpacArgs& A, int igs, double h) {
  const double wa = A.wlsub[igs - 1], wb = A.wlsub[igs];
  const double wl = 0.5 * (wa + wb);
  const double wlinv = 1.0 / wl;
  return 1.0 - exp(-(h * wlinv));
}

// Block: groups blockIdx.x * gpb + 1 .. + gpb one after another; warp w takes the
// 32 FS shells from (blockIdx.y * warps + w) 32 FS, lane l the FS from l FS on.
//
// Bound by instruction issue around the FP64 pipe: 11 FP64 operations per
// line-shell term (ten of them the exp), one shared-memory load, three integer
// operations for the exp and a line's and a row's share of loads and tests.
// FS shells per lane share a line record's load and index work; the warps of a
// block walk the same lines, so they share the records in L1 and end together;
// lines ordered by row leave one multiplication and one population load per row.
// Seven blocks per SM (72 registers) measured best of four to eight.  Whole builds
// in a loop on B200, before (lines in file order, four shells per lane, populations
// staged in shared memory, exp without the scaled argument and the spread table) and
// now: 4096 shells x 10000 groups x 2e6 lines 10.6 -> 9.65 ms, 256 x 2000 x 5e5 253 ->
// 173 us, 190 -> 134 where few ions are populated.
template <int FS>
__global__ void __launch_bounds__(kOpacWarps * 32, 7) opacity_fwd_kernel(const OpacArgs A, const ExpConst C, int gpb) {
  constexpr int FC = FS * OPAC_CT;
  extern __shared__ double etab[];  // kExpTabBytes
  exp_table_spread(etab);
  __syncthreads();
  const uint32_t mine = exp_table_mine();
  const int base = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * FC, lane = threadIdx.x & 31;
  if (base >= A.nc) return;  // uniform over the warp
  const int i0 = base + lane * FS;  // the lane's first shell (0-based)
  bool live[FS];
  double h[FS];
  ExpArg arg[FS];
  bool inrange = true;
#pragma unroll
  for (int s = 0; s < FS; ++s) {
    live[s] = i0 + s < A.nc && A.mass[i0 + s] > 0.0;
    // a shell that is not live runs the loops with h = 0 and is discarded
    h[s] = live[s] ? A.hckt[i0 + s] : 0.0;
    arg[s] = exp_arg(h[s]);
    inrange = inrange && h[s] >= 0.0 && h[s] * A.chimax <= 700.0;
  }
  // every exp argument -chi h of the warp's shells lies in [-700, 0]
  inrange = __all_sync(0xffffffffu, inrange);
  for (int ig = blockIdx.x * gpb + 1; ig <= min((int)(blockIdx.x + 1) * gpb, A.ng); ++ig) {
    double cap[FS], sp[FS], sr[FS];
#pragma unroll
    for (int s = 0; s < FS; ++s) cap[s] = sp[s] = sr[s] = 0.0;
    for (int g = 1; g <= A.ngs; ++g) {
      const int igs = (ig - 1) * A.ngs + g;
      double c[FS];
#pragma unroll
      for (int s = 0; s < FS; ++s) c[s] = 0.0;
      if (!A.nobb) {
        const int l0 = A.lstart[igs], n = A.lstart[igs + 1] - l0;
        if (n > 0) {
          // sum over the sub-group's lines of phi gxs ocg exp(-chilw h), times the
          // stimulated-emission factor once (the reference multiplies each term
          // by it; the sum of positive terms differs by rounding only)
          double sbb[FS];
          if (inrange) {
            bb_sums<FS>(A.lt + l0, n, arg, C, A.grndlev + i0, A.ld, etab, mine, sbb);
          } else {
#pragma unroll
            for (int s = 0; s < FS; ++s)
              sbb[s] = live[s] ? bb_sum_any(A.lt + l0, n, h[s], A.grndlev + i0 + s, A.ld) : 0.0;
          }
#pragma unroll
          for (int s = 0; s < FS; ++s)
            if (live[s]) c[s] = sbb[s] * kPgUnscale * bb_expfac(A, igs, h[s]);
        }
      }
      if (!A.nobf) {
        const BfTerm* t = A.bf + (size_t)(igs - 1) * A.maxbf;
        const int n = A.bnnz[igs - 1];
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
          const double2 v = __ldg(reinterpret_cast<const double2*>(t + k));
          double o[FS];
          load_run<FS>(A.ocp + i0 + (size_t)__double2loint(v.y) * A.ld, o);
#pragma unroll
          for (int s = 0; s < FS; ++s) c[s] = fma(v.x, o[s], c[s]);
        }
      }
      if (!A.noff) {
#pragma unroll
        for (int s = 0; s < FS; ++s)
          if (live[s]) c[s] = ff_add(A, i0 + s, igs, h[s], c[s]);
      }
#pragma unroll
      for (int s = 0; s < FS; ++s) {
        if (A.ngs == 1) cap[s] = c[s];
        else if (live[s] && c[s] > 0.0) { sp[s] = sp[s] + c[s]; sr[s] = sr[s] + 1.0 / c[s]; }
      }
    }
    if (A.ngs != 1) {
      // collapse subgridding, physical_opacity.f:252-264
      const double help = 1.0 / A.ngs;
#pragma unroll
      for (int s = 0; s < FS; ++s) {
        double capr = sr[s] * help;
        if (capr > 0.0) capr = 1.0 / capr;
        cap[s] = (1.0 - A.mix) * (sp[s] * help) + A.mix * capr;
      }
    }
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      const int i = i0 + s;
      if (i >= A.nc) continue;
      if (!live[s]) cap[s] = 0.0;
      const float c32 = (float)cap[s];
      float e32 = 0.f;
      if (live[s]) {
        const double wl = 0.5 * (A.grp_wl[ig] + A.grp_wl[ig - 1]);
        const double B_nu = (wl * wl / pc_c) * planck(wl, A.temp[i]);
        e32 = (float)(0.0 + cap[s] * B_nu);
        int f = 0;
        if (c32 == 0.f) f |= 1;
        if (c32 < 0.f) f |= 2;
        if (c32 != c32) f |= 4;
        if (c32 > FLT_MAX) f |= 8;
        if (f) atomicOr(A.flags, f);
      }
      // (ng, ncell): a shell's neighbouring groups are this block's next ones, so
      // the parts of a sector meet in L2
      const size_t o = (size_t)i * A.ng + (ig - 1);
      A.cap32[o] = c32;
      A.emiss32[o] = e32;
      if (A.capg64) A.capg64[o] = cap[s];
      if (A.cap64) A.cap64[(size_t)(ig - 1) * A.nc + i] = cap[s];
    }
  }
}

// ------------------------------------------------------------ analytic opacity
__global__ void analytic_opacity_kernel(int nc, int ng, const double* __restrict__ wlinv,
                                        const double* __restrict__ temp, const double* __restrict__ rho,
                                        int kind, double capcoef, double captpwr, double caprpwr,
                                        double sigcoef, double sigtpwr, double sigrpwr, double ldisp1,
                                        double ldisp2, double* __restrict__ sig, float* __restrict__ cap) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)nc * ng) return;
  const int i = (int)(t / ng), ig = (int)(t % ng) + 1;
  const double cc = capcoef * pow(temp[i], captpwr) * pow(rho[i], caprpwr);
  double v;
  if (kind == 1) v = cc;
  else if (kind == 2) {
    const double x1 = pc_hc * wlinv[ig] / pc_kb;
    const double x2 = pc_hc * wlinv[ig - 1] / pc_kb;
    v = 0.5 * cc * (x1 + x2) / sq(x1 * x2);
  } else {
    v = (ig % 2 == 1) ? cc * ldisp1 : cc * ldisp2;
  }
  cap[t] = (float)v;
  if (ig == 1) sig[i] = sigcoef * pow(temp[i], sigtpwr) * pow(rho[i], sigrpwr);
}

// ------------------------------------------------------------ Planck / Rosseland means
// Both integrals' weights from one exp, a fixed-shape tree reduction over groups.
// CT: float (gas_cap) or double (the FP64 opacity of the differentiable path),
// (ng, ncell).  With two exps per group and a reduction through nine block-wide
// steps: 90 us at 28800 shells x 100 groups (now 28), 303 us at 4096 x 10000 in
// FP64 (227).
template <class CT, int FORM>
__global__ void __launch_bounds__(256) opacity_means_kernel(int nc, int ng, const double* __restrict__ wlinv,
                                                            const double* __restrict__ temp,
                                                            const double* __restrict__ sig,
                                                            const CT* __restrict__ cap, double* __restrict__ capgrey,
                                                            double* __restrict__ capross) {
  constexpr int TPC = FORM == CELL_WARP ? 32 : 256;
  __shared__ double sh[2 * 8];
  __shared__ double part[FORM == CELL_BLOCK_WARP_ORDER ? 2 * kWarpCellGroups : 1];
  const int i = blockIdx.x * (256 / TPC) + threadIdx.x / TPC, t = threadIdx.x % TPC;
  if (i >= nc) return;  // uniform over the cell's threads
  const double tinv = 1.0 / temp[i];
  const double hct = hck * tinv;
  const double s = sig ? sig[i] : 0.0;
  auto add = [&](int g, double* a) {
    const double c = (double)cap[(size_t)i * ng + g];
    double w, wr;
    spec_weights(hct, wlinv, g, w, wr);
    a[0] = a[0] + c * w;
    a[1] = a[1] + (1.0 / (s + c)) * wr;
  };
  double a[2] = {0.0, 0.0};
  if (FORM == CELL_BLOCK_WARP_ORDER) {
    for (int g = t; g < ng; g += TPC) {
      double e[2] = {0.0, 0.0};
      add(g, e);
      part[g] = e[0];
      part[kWarpCellGroups + g] = e[1];
    }
    cell_sum_of_block<2>(part, kWarpCellGroups, ng, a, sh);
  } else {
    for (int g = t; g < ng; g += TPC) add(g, a);
    cell_sum<TPC, 2>(a, sh);
  }
  if (t == 0) {
    capgrey[i] = a[0];
    if (capross) capross[i] = 1.0 / a[1];
  }
}

// ------------------------------------------------------------ adjoint (no reference counterpart)
// specintv_elem and spectintv_elem of group g0 and their d/dT at temperature
// 1 / tinv (hct = hck tinv), from one exp and two divisions of the group's x:
// fplanck and fross and their derivatives in x, which are zero where the
// reference clamps x at 300; spectintv's NaN guard (groupmod.f:390-392) gives
// zero for both.  (Eight divisions: 526 us of means_bwd_kernel at 4096 x 10000, now 372.)
__device__ inline void spec_weights_dT(double hct, double tinv, const double* __restrict__ wlinv, int g0, double& w,
                                       double& wr, double& dw, double& dwr) {
  const double x1 = hct * wlinv[g0], x2 = hct * wlinv[g0 + 1];
  const double xm = 0.5 * (x2 + x1), ax = fabs(x2 - x1);
  double fp, fr, dfp, dfr;
  if (xm >= 300.0) {
    fp = fplanck(xm);
    fr = fross(xm);
    dfp = 0.0;
    dfr = 0.0;
  } else {
    const double ex = exp(xm), d = 1.0 / (ex - 1.0), exd = ex * d;
    fp = cube(xm) * d;
    fr = (pow4(xm) * d) * exd;
    dfp = (3.0 * sq(xm) - cube(xm) * exd) * d;
    const double v = fr * (4.0 / xm + 1.0 - 2.0 * exd);
    dfr = v != v ? 0.0 : v;
  }
  w = ftpi4 * ax * fp;
  dw = -(ftpi4 * ax * (fp + xm * dfp)) * tinv;
  const double sr = ftpi4r * ax * fr;
  const bool bad = sr != sr;  // groupmod.f:390-392
  wr = bad ? 0.0 : sr;
  dwr = bad ? 0.0 : -(ftpi4r * ax * (fr + xm * dfr)) * tinv;
}

// Adjoint of opacity_means_kernel<double>: adds to gcap (ng, ncell), gsig and gT.
__global__ void __launch_bounds__(256) means_bwd_kernel(int nc, int ng, const double* __restrict__ wlinv,
                                                        const double* __restrict__ temp,
                                                        const double* __restrict__ sig,
                                                        const double* __restrict__ cap,
                                                        const double* __restrict__ capross,
                                                        const double* __restrict__ ggrey,
                                                        const double* __restrict__ gross, double* __restrict__ gcap,
                                                        double* __restrict__ gsig, double* __restrict__ gT) {
  __shared__ double s1[256], s2[256];
  const int i = blockIdx.x;
  const double tinv = 1.0 / temp[i], hct = hck * tinv;
  const double s = sig[i];
  const double ug = ggrey ? ggrey[i] : 0.0;
  const double cr = capross[i];
  const double ur = gross ? gross[i] * cr * cr : 0.0;  // capross = 1/R: d capross = -capross^2 dR
  double asig = 0.0, at = 0.0;
  for (int g = threadIdx.x; g < ng; g += blockDim.x) {
    const double c = cap[(size_t)i * ng + g];
    double w, wr, dw, dwr;
    spec_weights_dT(hct, tinv, wlinv, g, w, wr, dw, dwr);
    const double inv = 1.0 / (s + c);
    const double dr = wr * inv * inv;  // -dR/dc
    gcap[(size_t)i * ng + g] += ug * w + ur * dr;
    asig = asig + ur * dr;
    at = at + ug * c * dw - ur * inv * dwr;
  }
  s1[threadIdx.x] = asig;
  s2[threadIdx.x] = at;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      s1[threadIdx.x] += s1[threadIdx.x + w];
      s2[threadIdx.x] += s2[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    gsig[i] += s1[0];
    gT[i] += s2[0];
  }
}

struct OpacBwd {
  const double* gcap;  // (ng, ncell)
  double* gT;          // (ncell), added to
  double* ggrnd;       // [slot][cell], added to (d cap / d grndlev)
  double* goc;         // [slot][cell], added to (bound-free)
  double* ghlp;        // (ncell), added to (d cap / d hlparr)
  double* gfr;         // (0:nelem, ncell), added to
};

// The bound-bound part of the adjoint of one group for FS shells of a lane (i0,
// i0 + 32 ...; ue: dL/dcap times the stimulated-emission factor): adds ue * pg *
// exp(-chi h) of every line (d cap / d grndlev) to dL/d grndlev of its row, the
// row's sum by one reduction without return (coalesced over the warp's shells),
// and returns the sums over lines of pg exp(-chi h) og (capbb over that factor)
// and of the same times chi (the T-derivative's weight).  FAST: exp_scaled's
// range holds for every argument.
template <int FS, bool FAST>
__device__ __forceinline__ void bb_adjoint(const LineTerm* __restrict__ lt, int n, const double* h, const ExpArg* arg,
                                           const ExpConst& C, const double* ue, const double* __restrict__ pop, int ld,
                                           double* __restrict__ ggrnd, int nc, const double* s_tab, uint32_t mine,
                                           double* sbb, double* schi) {
  double og[FS];
  auto row_begin = [&](unsigned idx) {
    const double* g = pop + (size_t)line_row(idx) * ld;
#pragma unroll
    for (int s = 0; s < FS; ++s) og[s] = __ldg(g + s * OPAC_CT);
  };
  auto term = [&](const LineVals& v, double* acc, double* accc) {
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      const double e = v.pg * (FAST ? exp_scaled(v.chi, arg[s], C, s_tab, mine) : exp(-(v.chi * h[s])));
      acc[s] = acc[s] + e;
      accc[s] = fma(e, v.chi, accc[s]);
    }
  };
  LineVals t = load_line(lt);
  row_begin(t.idx);
#pragma unroll
  for (int s = 0; s < FS; ++s) sbb[s] = schi[s] = 0.0;
  const LineTerm* const end = lt + n;
  do {
    double acc[FS], accc[FS];
#pragma unroll
    for (int s = 0; s < FS; ++s) acc[s] = accc[s] = 0.0;
    const int slot = line_slot(t.idx);
#pragma unroll 1
    for (;;) {
      const LineVals u = load_line(lt + 1);
      term(t, acc, accc);
      ++lt;
      if (t.idx & kLineRowEnd) {  // the same for the whole warp
        t = u;
        break;
      }
      t = load_line(lt + 1);
      term(u, acc, accc);
      ++lt;
      if (u.idx & kLineRowEnd) break;
    }
    double* g = ggrnd + (size_t)slot * nc;
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      if (ue[s] != 0.0) atomicAdd(g + s * OPAC_CT, ue[s] * acc[s]);
      sbb[s] = fma(acc[s], og[s], sbb[s]);
      schi[s] = fma(accc[s], og[s], schi[s]);
    }
    row_begin(t.idx);  // (any row's where none follows)
  } while (lt < end);
}

// Adjoint of the forward's groups (ngs = 1), bound-bound part: one pass over the
// lines of each group (bf: bf_bwd_kernel, ff: ff_bwd_kernel).  Block: groups blockIdx.x * gpb + 1 .. + gpb
// one after another; warp w takes the 32 FS shells from (blockIdx.y * warps + w)
// 32 FS, lane l shells l, l + 32 ... of them.  Bound like the forward, with 13
// FP64 operations per term; a population row's gradient leaves by one
// reduction per (row, group) instead of one per line, whose L2 traffic held the
// kernel at half its arithmetic's rate.
template <int FS>
__global__ void __launch_bounds__(kOpacWarps * 32, 5) opacity_bwd_kernel(const OpacArgs A, const OpacBwd B,
                                                                               const ExpConst C, int gpb) {
  __shared__ double etab[kExpTabN * kExpCopies];
  exp_table_spread(etab);
  __syncthreads();
  const uint32_t mine = exp_table_mine();
  const int base = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (FS * OPAC_CT), lane = threadIdx.x & 31;
  if (base >= A.nc) return;  // uniform over the warp
  bool live[FS];
  int ii[FS];
  double h[FS], gt[FS];
  ExpArg arg[FS];
  bool inrange = true;
#pragma unroll
  for (int s = 0; s < FS; ++s) {
    const int i = base + s * OPAC_CT + lane;
    ii[s] = min(i, A.nc - 1);
    live[s] = i < A.nc && A.mass[ii[s]] > 0.0;
    h[s] = live[s] ? A.hckt[ii[s]] : 0.0;
    arg[s] = exp_arg(h[s]);
    inrange = inrange && h[s] >= 0.0 && h[s] * A.chimax <= 700.0;  // as in the forward
    gt[s] = 0.0;
  }
  inrange = __all_sync(0xffffffffu, inrange);
  const double* const pop = A.grndlev + base + lane;
  for (int ig = blockIdx.x * gpb + 1; ig <= min((int)(blockIdx.x + 1) * gpb, A.ng); ++ig) {
    double u[FS];
    bool any = false;
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      u[s] = live[s] ? B.gcap[(size_t)ii[s] * A.ng + (ig - 1)] : 0.0;
      any = any || u[s] != 0.0;
    }
    if (!__any_sync(0xffffffffu, any)) continue;
    const int l0 = A.lstart[ig], n = A.lstart[ig + 1] - l0;
    if (n <= 0) continue;
    const double wa = A.wlsub[ig - 1], wb = A.wlsub[ig];
    const double wl = 0.5 * (wa + wb);
    const double wlinv = 1.0 / wl;
    double eh[FS], ue[FS], sbb[FS], schi[FS];
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      eh[s] = exp(-(h[s] * wlinv));
      ue[s] = u[s] != 0.0 ? u[s] * (1.0 - eh[s]) * kPgUnscale : 0.0;  // (a term's pg has kPgScale)
    }
    if (inrange)
      bb_adjoint<FS, true>(A.lt + l0, n, h, arg, C, ue, pop, A.ld, B.ggrnd + ii[0], A.nc, etab, mine, sbb,
                           schi);
    else
      bb_adjoint<FS, false>(A.lt + l0, n, h, arg, C, ue, pop, A.ld, B.ggrnd + ii[0], A.nc, etab, mine,
                            sbb, schi);
#pragma unroll
    for (int s = 0; s < FS; ++s) {
      if (u[s] == 0.0) continue;
      sbb[s] *= kPgUnscale;
      schi[s] *= kPgUnscale;
      const double expfac = 1.0 - eh[s], T = A.temp[ii[s]];
      // h = hc/kT: d exp(-chi h)/dT = chi h/T exp(..), d expfac/dT = -(h/T) wlinv eh
      gt[s] = gt[s] + u[s] * ((h[s] / T) * (schi[s] * expfac) - sbb[s] * expfac * (h[s] / T) * wlinv * eh[s] / expfac);
    }
  }
#pragma unroll
  for (int s = 0; s < FS; ++s)
    if (gt[s] != 0.0) atomicAdd(&B.gT[ii[s]], gt[s]);
}

// Free-free part of the adjoint (physical_opacity.f:197-247, ngs = 1).  The
// shell's opacity at a group is hn hlparr sum_z z^2 fr_z gff_z, gff_z linear in
// two rows of the table (the group's iu, du) between two columns (the shell's
// igg, dgg of the element).  A block takes one shell, a warp 64 consecutive
// groups at a time, a lane two of them:
// - elements without the gff >= 1 clamp: d cap / d fr(z) = help z^2 gff_z, so
//   sum_g u_g help_g gff_z = sum_j W[j] Gz[j] with W[j] the groups' row weights
//   times u help (u = dL/dcap).  Neighbouring groups share their row (a decade of
//   wavelengths is ten rows), so a warp adds one pair of sums per distinct row
//   to W; dL/dT from the shell's sums over elements (opac_cell_kernel);
// - clamped elements, the same for the whole block: one by one, a sum over the
//   warp each.
// All that depends on the shell, and nearly always the table's row, is the same
// for the whole warp, and gcap is read along the groups.  With a shell per lane
// at the end of each of opacity_bwd_kernel's groups, it read the table and gcap
// with a sector per lane, added to W in memory twice per (shell, group) and held
// registers that the line loop wanted: 4.1 of the adjoint's 16.4 ms at 4096 x 10000
// (now 1.4), and another 25 us in a kernel for the products with W.  Bound by FP64
// issue (log10, exp, three divisions and the clamped elements per pair).  One or four
// groups a lane, or blocks of four warps: 0.05 to 0.2 ms more.
constexpr int kFfK = 2, kFfWarps = 8;
__global__ void __launch_bounds__(kFfWarps * 32) ff_bwd_kernel(const OpacArgs A, const OpacBwd B) {
  __shared__ double sW[kFfWarps][FF_NU];
  __shared__ double sfr[kFfWarps][32];
  __shared__ double sg[2][kFfWarps];
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  if (!(A.mass[i] > 0.0)) return;  // uniform over the block
  for (int j = lane; j < FF_NU; j += 32) sW[warp][j] = 0.0;
  sfr[warp][lane] = 0.0;
  __syncwarp();
  const double T = A.temp[i], h = A.hckt[i], hl = A.hlparr[i];
  const double ln10 = 2.302585092994045684;
  const double dru = -10.0 / (ln10 * T), drgg = -5.0 / (ln10 * T);  // table coordinates vs T
  const double* Sv = A.ffsum + (size_t)i * FF_NU;
  const double* Dv = A.ffdsum + (size_t)i * FF_NU;
  const double* nfr = A.natomfr + (size_t)(A.nelem + 1) * i;
  const double* G = A.gff;
  const unsigned clamped = A.ffclamp_all[i];
  double a[2] = {0.0, 0.0};  // dL/dT, dL/d hlparr
  for (int g0 = (blockIdx.y * nwarp + warp) * (32 * kFfK); g0 < A.ng; g0 += gridDim.y * nwarp * (32 * kFfK)) {
    int iu[kFfK];  // 0: nothing to do
    double u[kFfK], hn[kFfK], du[kFfK], dlnhelp[kFfK], S[kFfK], dS[kFfK];
#pragma unroll
    for (int k = 0; k < kFfK; ++k) {
      const int ig = g0 + 32 * k + lane;
      iu[k] = 0;
      u[k] = ig < A.ng ? B.gcap[(size_t)i * A.ng + ig] : 0.0;
      if (u[k] == 0.0) continue;
      const double wl = A.wlsub[ig];
      const double wlinv = 1.0 / wl;
      const double uu = h * wlinv;
      const double ru = 10.0 * (log10(uu) + 4.0) + 1.0;
      iu[k] = !(ru >= 1.0) ? 1 : (ru >= (double)(FF_NU - 1) ? FF_NU - 1 : (int)floor(ru));
      du[k] = ru - iu[k];
      const double eu = exp(-uu);
      hn[k] = A.ffc1 * sqrt(h) * (1.0 - eu) * cube(wl);
      dlnhelp[k] = -0.5 / T - eu * uu / (T * (1.0 - eu));
      // unclamped elements: S = sum z^2 fr gff, dS/dT through the table row (du) and
      // column (dgg)
      const double s0 = Sv[iu[k] - 1], s1 = Sv[iu[k]];
      S[k] = (1.0 - du[k]) * s0 + du[k] * s1;
      dS[k] = (s1 - s0) * dru + ((1.0 - du[k]) * Dv[iu[k] - 1] + du[k] * Dv[iu[k]]) * drgg;
    }
    // elements under the gff >= 1 clamp
    for (unsigned m = clamped; m; m &= m - 1) {
      const int iz = __ffs(m);
      const double fr = nfr[iz];
      const int igg = -A.ffigg[(size_t)(iz - 1) * A.nc + i];
      const double dgg = A.ffdgg[(size_t)(iz - 1) * A.nc + i];
      const double w = (double)(iz * iz);
      double v[1] = {0.0};
#pragma unroll
      for (int k = 0; k < kFfK; ++k) {
        if (iu[k] == 0) continue;
        // the table's rows iu - 1 and iu at the element's column, and their slopes over it
        const double* q = G + (iu[k] - 1) + FF_NU * (igg - 1);
        const double g00 = q[0], g10 = q[1], c0 = q[FF_NU] - g00, c1 = q[FF_NU + 1] - g10;
        const double r0 = g00 + dgg * c0, dr = (g10 + dgg * c1) - r0;
        const double graw = r0 + du[k] * dr;
        const bool flat = graw < 1.0;
        const double g = flat ? 1.0 : graw;
        const double dg = flat ? 0.0 : dr * dru + (c0 + du[k] * (c1 - c0)) * drgg;
        v[0] = v[0] + u[k] * (hn[k] * hl) * g * w;
        if (fr == 0.0) continue;
        S[k] = S[k] + g * w * fr;
        dS[k] = dS[k] + dg * w * fr;
      }
      cell_sum<32, 1>(v, nullptr);
      if (lane == 0) sfr[warp][iz - 1] = sfr[warp][iz - 1] + v[0];
    }
#pragma unroll
    for (int k = 0; k < kFfK; ++k) {
      if (iu[k] == 0) continue;
      const double help = hn[k] * hl;
      a[0] = a[0] + u[k] * (help * S[k] * dlnhelp[k] + help * dS[k]);
      a[1] = a[1] + u[k] * hn[k] * S[k];
      u[k] = u[k] * help;
    }
    // the unclamped elements' row weights
    for (;;) {
      int j = FF_NU;
#pragma unroll
      for (int k = 0; k < kFfK; ++k)
        if (iu[k] != 0) j = min(j, iu[k]);
      j = __reduce_min_sync(0xffffffffu, j);
      if (j == FF_NU) break;  // iu < FF_NU
      double v[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < kFfK; ++k) {
        if (iu[k] != j) continue;
        v[0] = v[0] + u[k] * (1.0 - du[k]);
        v[1] = v[1] + u[k] * du[k];
        iu[k] = 0;
      }
      cell_sum<32, 2>(v, nullptr);
      if (lane == 0) {
        sW[warp][j - 1] = sW[warp][j - 1] + v[0];
        sW[warp][j] = sW[warp][j] + v[1];
      }
    }
  }
  cell_sum<32, 2>(a, nullptr);
  if (lane == 0) {
    sg[0][warp] = a[0];
    sg[1][warp] = a[1];
  }
  // the block's sums, and the product of W with the elements' columns, eight
  // lanes an element
  __syncthreads();
  for (int j = threadIdx.x; j < FF_NU; j += blockDim.x) {
    double w = sW[0][j];
    for (int k = 1; k < nwarp; ++k) w = w + sW[k][j];
    sW[0][j] = w;
  }
  if (threadIdx.x < 2) {
    double w = sg[threadIdx.x][0];
    for (int k = 1; k < nwarp; ++k) w = w + sg[threadIdx.x][k];
    if (w != 0.0) atomicAdd((threadIdx.x ? B.ghlp : B.gT) + i, w);
  }
  __syncthreads();
  for (int z0 = 0; z0 < A.nelem; z0 += blockDim.x >> 3) {
    const int z = z0 + (threadIdx.x >> 3), t = threadIdx.x & 7;  // element z + 1
    const bool some = z < A.nelem;
    double acc = 0.0;
    if (some && (clamped >> z & 1u)) {
      for (int k = t; k < nwarp; k += 8) acc = acc + sfr[k][z];
    } else if (some) {
      const int igg = A.ffigg[(size_t)z * A.nc + i];
      const double dgg = A.ffdgg[(size_t)z * A.nc + i];
      for (int j = t; j < FF_NU; j += 8)
        if (sW[0][j] != 0.0)  // (most rows lie outside the groups' range)
          acc = acc + sW[0][j] * ((1.0 - dgg) * G[j + FF_NU * (igg - 1)] + dgg * G[j + FF_NU * igg]);
      acc = (double)((z + 1) * (z + 1)) * acc;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) acc = acc + __shfl_xor_sync(0xffffffffu, acc, o);
    if (some && t == 0) atomicAdd(&B.gfr[(size_t)i * (A.nelem + 1) + z + 1], acc);
  }
}

// Bound-free part of the adjoint (physical_opacity.f:163-195, ngs = 1):
// d cap(g, i) / d oc(slot, i) = xs(g, slot) mbarn, so
// goc(act_slot(a), i) += mbarn sum_g gcap(g, i) xs(g, a) over the active slots a
// -- a product of the (shell, group) gradient with the (group, slot) table.
// Tiled like a matrix product: a block computes 32 shells x 32 slots, staging
// 32 groups of both operands in shared memory per round; thread (tx, ty)
// holds shell tx and slots ty, ty + 8, ty + 16, ty + 24.  The groups are split
// over gridDim.z blocks, whose parts are added by atomics: on small grids a
// block per (32 shells, 32 slots) left most SMs idle (256 x 2000: 72 blocks, 165
// us; split
// 21 us; 4096 x 10000: 737 -> 415 us).  Runs after opacity_bwd_kernel and before
// opac_cell_bwd_kernel.
constexpr int BFB_T = 32;
__global__ void __launch_bounds__(BFB_T * 8) bf_bwd_kernel(const OpacArgs A, const OpacBwd B) {
  __shared__ double su[BFB_T][BFB_T + 1];  // [shell][group]
  __shared__ double sx[BFB_T][BFB_T + 1];  // [group][slot]
  const int nact = *A.pnact;
  const int a0 = blockIdx.y * BFB_T;
  if (a0 >= nact) return;  // uniform over the block
  const int i0 = blockIdx.x * BFB_T;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const int ntile = (A.ng + BFB_T - 1) / BFB_T;
  const int t0 = (int)((long long)ntile * blockIdx.z / gridDim.z), t1 = (int)((long long)ntile * (blockIdx.z + 1) / gridDim.z);
  for (int g0 = t0 * BFB_T; g0 < t1 * BFB_T; g0 += BFB_T) {
    // the cross sections first: most (group, slot) tiles lie beyond the slots'
    // ionisation edges, all zero, and are skipped (the forward skips xs = 0)
    bool nz = false;
    for (int k = threadIdx.x; k < BFB_T * BFB_T; k += blockDim.x) {
      const int r = k >> 5, q = k & 31;  // sx: group r, slot q
      const int gr = g0 + r, a = a0 + q;
      const double x = (gr < A.ng && a < nact) ? A.xstab[(size_t)gr * A.maxact + A.act_slot[a]] : 0.0;
      sx[r][q] = x;
      nz = nz || x != 0.0;
    }
    if (!__syncthreads_or(nz)) continue;  // block-uniform
    for (int k = threadIdx.x; k < BFB_T * BFB_T; k += blockDim.x) {
      const int r = k >> 5, q = k & 31;  // su: shell r, group q (coalesced over groups)
      const int ii = i0 + r, g = g0 + q;
      su[r][q] = (ii < A.nc && g < A.ng) ? B.gcap[(size_t)ii * A.ng + g] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < BFB_T; ++q) {
      const double u = su[tx][q];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = acc[j] + u * sx[q][ty + 8 * j];
    }
    __syncthreads();
  }
  const int i = i0 + tx;
  if (i >= A.nc || !(A.mass[i] > 0.0)) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int a = a0 + ty + 8 * j;
    if (a < nact && acc[j] != 0.0) atomicAdd(&B.goc[(size_t)A.act_slot[a] * A.nc + i], acc[j]);  // xstab holds * pc_mbarn
  }
}

// Adjoint of opac_cell_kernel: grndlev = oc ginv, hlparr = (natom/vol)^2
// nelec, gas_sig = cthomson nelec natom / vol.
__global__ void opac_cell_bwd_kernel(int nc, int nelem, int nst, const int32_t* __restrict__ ion_ni,
                                     const double* __restrict__ natom, const double* __restrict__ nelec,
                                     const double* __restrict__ vol, const double* __restrict__ mass,
                                     const double* __restrict__ ginv, int nothmson,
                                     const double* __restrict__ ggrnd, const double* __restrict__ ghlp,
                                     const double* __restrict__ gsig, double* __restrict__ goc,
                                     double* __restrict__ gnelec, double* __restrict__ gnatom) {
  // one thread per (shell i, element iz = blockIdx.y + 1); element 1's threads
  // also write the shell's scalars
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  if (!(mass[i] > 0.0)) {
    if (blockIdx.y == 0) {
      gnelec[i] = 0.0;
      gnatom[i] = 0.0;
    }
    return;
  }
  {
    const int iz = blockIdx.y + 1;
    const int lim = min(iz, ion_ni[iz - 1] - 1);
    for (int ii = 1; ii <= lim && ii <= nst; ++ii) {
      const size_t k = ((size_t)(iz - 1) * nst + (ii - 1)) * nc + i;
      goc[k] += ggrnd[k] * ginv[k];
    }
  }
  if (blockIdx.y != 0) return;
  const double nd = natom[i] / vol[i];
  double gne = ghlp[i] * nd * nd;
  double gna = ghlp[i] * 2.0 * nd * nelec[i] / vol[i];
  if (!nothmson) {
    gne += gsig[i] * cthomson * natom[i] / vol[i];
    gna += gsig[i] * cthomson * nelec[i] / vol[i];
  }
  gnelec[i] = gne;
  gnatom[i] = gna;
}

}  // namespace

// ============================================================ launchers
// Groups that a block of the line kernels takes one after another: one, except on
// the largest grids, where more save filling the exp table (warps: of two shells
// per lane over all groups).  Measured on B200, one against `most` groups: forward
// 4096 x 10000 (640000 warps) 5.37 against 5.30 ms, 10000 x 1000 (157000) 1.34
// against 1.36, 1024 x 500 248 against 311 us, 1024 x 64 240 against 847 us, whose
// grid then leaves the chip idle; adjoint 9.62 against 9.10 ms, 4096 x 2000 (128000)
// 3.12 against 3.22, 1024 x 64 345 against 1621 us (whole calls).
static int groups_per_block(int nc, int ng, int most) {
  const long long warps = (long long)ng * ((nc + 2 * OPAC_CT - 1) / (2 * OPAC_CT));
  return warps >= 400000 ? most : 1;
}

// One launch of opacity_fwd_kernel on the stream.  One shell per lane where two
// would leave lanes without a shell, or less than three warps for a scheduler:
// with so few, the chain of a warp's lines is what counts, and it is shorter with
// one exp a line.  Measured on B200, whole calls with one / two shells per lane:
// 128 shells x 20 groups (40 warps of two) 542 / 661 us, 1024 x 64 (1024) 203 /
// 240, 256 x 500 (2000) 103 / 95, 512 x 300 (2400) 187 / 166, 256 x 2000 196 / 175;
// 96 x 10000 186 / 199 and 97 x 10000 230 / 197 (a fourth of two shells' lanes idle,
// none); 77 x 333 of three sub-groups 16 / 19.  Four shells hold too many registers
// for the warps they leave (256 x 2000 214 against 178 us, 4096 x 10000 9.23 against
// 8.86 ms).
static int launch_fwd(slg_ctx* ctx, OpacArgs& A) {
  const int t1 = (A.nc + OPAC_CT - 1) / OPAC_CT, t2 = (t1 + 1) / 2;
  const bool fill = (long long)A.ng * t2 >= 3LL * 4 * ctx->num_sms;
  const int fs = fill && t1 != 1 && t1 != 3 ? 2 : 1;
  const int tiles = fs == 2 ? t2 : t1, warps = tiles < kOpacWarps ? tiles : kOpacWarps;
  const int gpb = groups_per_block(A.nc, A.ng, 4);
  const dim3 grid((A.ng + gpb - 1) / gpb, (tiles + warps - 1) / warps);
  if (fs == 2) opacity_fwd_kernel<2><<<grid, warps * 32, kExpTabBytes, ctx->stream>>>(A, ExpConst{}, gpb);
  else opacity_fwd_kernel<1><<<grid, warps * 32, kExpTabBytes, ctx->stream>>>(A, ExpConst{}, gpb);
  return cuda_check(ctx, cudaGetLastError(), "opacity_fwd launch");
}

// What the build needs of the groups, the line list and the bound-free fits
// alone, for ngs sub-groups per group: laid out on the first call after
// slg_set_groups or slg_set_atomic_data (or for another ngs) and kept, like the
// atomic data, until the next.  While a graph is being captured or held the
// layout is queued with every call, so that each graph lays out what its own
// calls read.
static int opacity_plan(slg_ctx* ctx, int ngs, bool need_bb, bool need_bf, OpacArgs& A) {
  const int ngsub = ctx->ng * ngs, nslot = ctx->nelem * ctx->nstage, nst = ctx->nstage;
  const int nedge = ngsub + 1, nedge_pad = (nedge + 1) & ~1;
  cudaStream_t st = ctx->stream;
  if (ctx->plan_ngs != ngs) ctx->plan_edges = ctx->plan_bb = ctx->plan_bf = false;
  const bool keep = !ctx->capturing && !ctx->graph_exec;
  if (!keep) ctx->plan_edges = ctx->plan_bb = ctx->plan_bf = false;
  double* d_wlsub = (double*)scratch(ctx, 0, sizeof(double) * nedge_pad);
  if (!d_wlsub) return SLG_ERR_OOM;
  if (!ctx->plan_edges)
    wlsub_kernel<<<(nedge_pad + 255) / 256, 256, 0, st>>>(ctx->ng, ngs, nedge_pad, ctx->d_wl, d_wlsub);
  A.wlsub = d_wlsub;
  A.lstart = nullptr;
  A.lt = nullptr;
  if (need_bb) {
    if (ngsub > kMaxLineSubgroups)
      return set_error(ctx, SLG_ERR_ARG, "too many sub-groups for line binning (%d)", ngsub);
    int* d_lstart = (int*)scratch(ctx, 2, sizeof(int) * (nedge + 3));
    // one record past the last is loaded ahead
    LineTerm* d_lt = (LineTerm*)scratch(ctx, 84, sizeof(LineTerm) * ((size_t)ctx->nline + 2));
    if (!d_lstart || !d_lt) return SLG_ERR_OOM;
    if (!ctx->plan_bb) {
      line_range_kernel<<<(nedge + 2 + 127) / 128, 128, 0, st>>>(ctx->d_bb, ctx->nline, d_wlsub, nedge, d_lstart);
      // lines outside the groups, and past the last, are never used but may be loaded
      cudaMemsetAsync(d_lt, 0, sizeof(LineTerm) * ((size_t)ctx->nline + 2), st);
      const size_t shm = sizeof(int) * LT_WARPS * (size_t)ctx->nlrow;  // at most 30 x 64 rows: 30 KB
      line_terms_kernel<<<(ngsub + LT_WARPS - 1) / LT_WARPS, LT_WARPS * 32, shm, st>>>(
          ctx->d_bb, d_lstart, ngsub, d_wlsub, nst, ctx->d_lrow_of_slot, ctx->nlrow, d_lt);
    }
    A.lstart = d_lstart;
    A.lt = d_lt;
  }
  A.xstab = nullptr;
  if (need_bf) {
    const size_t n = (size_t)ngsub * nslot;
    double* d_xs = (double*)scratch(ctx, 11, sizeof(double) * n);
    if (!d_xs) return SLG_ERR_OOM;
    if (!ctx->plan_bf)
      bf_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ngsub, nslot, ctx->d_ion_ni, nst, d_wlsub,
                                                                   ctx->d_ph1, ctx->d_ph2, d_xs);
    A.xstab = d_xs;
  }
  const int rc = cuda_check(ctx, cudaGetLastError(), "opacity plan launch");
  if (!rc && keep) {
    ctx->plan_ngs = ngs;
    ctx->plan_edges = true;
    ctx->plan_bb = ctx->plan_bb || need_bb;
    ctx->plan_bf = ctx->plan_bf || need_bf;
  }
  return rc;
}

// Everything the opacity kernels read, queued on the stream: the plan, the
// per-cell terms (and gas_sig) and the populated ions' bound-free terms.
static int opacity_prepare(slg_ctx* ctx, const slg_gas* gas, const slg_opacity_flags* flags, double* gas_sig,
                           OpacArgs& A) {
  const int nc = ctx->nx, ng = ctx->ng;
  const int ngs = flags->ngs < 1 ? 1 : flags->ngs;
  const int ngsub = ng * ngs;
  const int nelem = ctx->nelem, nst = ctx->nstage;
  const int nslot = nelem * nst;
  cudaStream_t st = ctx->stream;
  if (nelem <= 0) return set_error(ctx, SLG_ERR_STATE, "atomic data not set");
  const bool do_bb = ctx->nline > 0 && !flags->nobb, do_bf = !flags->nobf;
  const bool do_ff = !flags->noff && ctx->d_gff;
  int rc = opacity_plan(ctx, ngs, do_bb, do_bf, A);
  if (rc) return rc;
  int* d_flags = (int*)scratch(ctx, 3, sizeof(int) * (4 + nslot));  // sanity word, then the active slots
  double* d_hckt = (double*)scratch(ctx, 4, sizeof(double) * nc);
  double* d_hlp = (double*)scratch(ctx, 5, sizeof(double) * nc);
  const int ld = padded_shells(nc), nrow = ctx->nlrow;
  double* d_ocp = (double*)scratch(ctx, 6, sizeof(double) * (size_t)ld * (nslot + nrow));
  double* d_grnd = d_ocp + (size_t)ld * nslot;
  int* d_ffigg = (int*)scratch(ctx, 7, sizeof(int) * (size_t)nc * nelem);
  double* d_ffdgg = (double*)scratch(ctx, 8, sizeof(double) * (size_t)nc * nelem);
  double* d_ffsum = (double*)scratch(ctx, 88, sizeof(double) * 2 * (size_t)nc * FF_NU);
  unsigned* d_ffclamp = (unsigned*)scratch(ctx, 89, sizeof(unsigned) * 2 * (size_t)nc);
  if (!d_flags || !d_hckt || !d_hlp || !d_ocp || !d_ffigg || !d_ffdgg || !d_ffsum || !d_ffclamp) return SLG_ERR_OOM;
  int* d_active = d_flags + 4;
  cudaMemsetAsync(d_flags, 0, sizeof(int) * (4 + nslot), st);
  double* d_ffdsum = d_ffsum + (size_t)nc * FF_NU;
  opac_cell_kernel<<<(ld + CELLS - 1) / CELLS, CELLS * 32, 0, st>>>(
      nc, nelem, nst, ctx->d_ion_ni, gas->temp, gas->natom, gas->nelec, gas->vol, gas->mass, gas->oc, gas->ginv,
      flags->nothmson, gas->natomfr, do_ff ? ctx->d_gff : nullptr, d_hckt, gas_sig, d_hlp, ld,
      do_bb ? nrow : 0, ctx->d_lrow_of_slot + nslot, d_grnd, d_ocp, d_active, d_ffigg, d_ffdgg, d_ffsum, d_ffdsum,
      d_ffclamp, d_ffclamp + nc);
  if (do_bf) {
    A.maxbf = 0;
    for (int z = 1; z <= nelem; ++z) A.maxbf += std::max(0, std::min(std::min(z, ctx->h_ion_ni[z - 1] - 1), nst));
    BfTerm* d_bf = (BfTerm*)scratch(ctx, 86, sizeof(BfTerm) * (size_t)ngsub * A.maxbf);
    int* d_bnnz = (int*)scratch(ctx, 87, sizeof(int) * (size_t)ngsub);
    if (!d_bf || !d_bnnz) return SLG_ERR_OOM;
    bf_select_kernel<<<(ngsub + 7) / 8, 256, 0, st>>>(ngsub, nslot, A.maxbf, A.xstab, d_active, d_bf, d_bnnz);
    A.bf = d_bf;
    A.bnnz = d_bnnz;
  }
  A.nc = nc; A.ng = ng; A.ngs = ngs; A.ngsub = ngsub; A.nelem = nelem; A.nst = nst; A.maxact = nslot;
  A.pnact = nullptr;
  A.nobb = !do_bb; A.nobf = !do_bf; A.noff = flags->noff;
  A.mix = flags->opacmixrossel;
  A.grp_wl = ctx->d_wl;
  A.chimax = ctx->line_chimax;
  A.ld = ld; A.ocp = d_ocp;
  A.grndlev = d_grnd; A.active = d_active; A.act_slot = nullptr;
  A.hckt = d_hckt; A.hlparr = d_hlp; A.mass = gas->mass; A.natomfr = gas->natomfr; A.temp = gas->temp;
  A.ffigg = d_ffigg; A.ffdgg = d_ffdgg; A.gff = ctx->d_gff;
  A.ffsum = d_ffsum; A.ffdsum = d_ffdsum; A.ffclamp = d_ffclamp; A.ffclamp_all = d_ffclamp + nc;
  A.ffc1 = ff_c1a * sqrt(ff_c1b);
  A.cap32 = nullptr; A.emiss32 = nullptr; A.cap64 = nullptr; A.capg64 = nullptr; A.flags = d_flags;
  if (!ctx->d_gff && !A.noff) return set_error(ctx, SLG_ERR_STATE, "free-free table not set");
  return cuda_check(ctx, cudaGetLastError(), "opacity preparation launch");
}

int launch_physical_opacity(slg_ctx* ctx, const slg_gas* gas, const slg_opacity_flags* flags,
                            double* gas_sig, float* gas_cap, float* gas_emiss, double* cap64) {
  OpacArgs A;
  const int rc = opacity_prepare(ctx, gas, flags, gas_sig, A);
  if (rc) return rc;
  A.cap32 = gas_cap; A.emiss32 = gas_emiss; A.cap64 = cap64;
  return launch_fwd(ctx, A);
}

// Physical opacity (ngs = 1) with the FP64 result in gas_cap's (ng, ncell)
// layout; gas_cap/gas_emiss (float) are written as well.
int launch_physical_opacity64(slg_ctx* ctx, const slg_gas* gas, double* gas_sig, double* capg64, float* gas_cap,
                              float* gas_emiss) {
  slg_opacity_flags fl{0, 0, 0, 0, 1, 0.0};
  OpacArgs A;
  const int rc = opacity_prepare(ctx, gas, &fl, gas_sig, A);
  if (rc) return rc;
  A.cap32 = gas_cap; A.emiss32 = gas_emiss; A.capg64 = capg64;
  return launch_fwd(ctx, A);
}

template <class CT>
static void launch_means(slg_ctx* ctx, const double* temp, const double* sig, const CT* cap, double* capgrey,
                         double* capross) {
  const int nc = ctx->nx, ng = ctx->ng;
  const CellForm form = cell_form(nc, ng, ctx->num_sms);
  const int nblk = form == CELL_WARP ? (nc + 7) / 8 : nc;
  auto* kernel = form == CELL_WARP               ? opacity_means_kernel<CT, CELL_WARP>
                 : form == CELL_BLOCK_WARP_ORDER ? opacity_means_kernel<CT, CELL_BLOCK_WARP_ORDER>
                                                 : opacity_means_kernel<CT, CELL_BLOCK>;
  kernel<<<nblk, 256, 0, ctx->stream>>>(nc, ng, ctx->d_wlinv, temp, sig, cap, capgrey, capross);
}

int launch_opacity_means64(slg_ctx* ctx, const double* temp, const double* sig, const double* cap,
                           double* capgrey, double* capross) {
  launch_means(ctx, temp, sig, cap, capgrey, capross);
  return cuda_check(ctx, cudaGetLastError(), "opacity_means64 launch");
}

int launch_means_bwd(slg_ctx* ctx, const double* temp, const double* sig, const double* cap, const double* capross,
                     const double* ggrey, const double* gross, double* gcap, double* gsig, double* gT) {
  means_bwd_kernel<<<ctx->nx, 256, 0, ctx->stream>>>(ctx->nx, ctx->ng, ctx->d_wlinv, temp, sig, cap, capross, ggrey,
                                                    gross, gcap, gsig, gT);
  return cuda_check(ctx, cudaGetLastError(), "means adjoint launch");
}

// Adjoint of launch_physical_opacity64 for gcap (ng, ncell) and gsig: adds
// dL/dT to gT and writes dL/d(oc, nelec, natom, natomfr) (goc [slot][cell],
// gnelec, gnatom, gfr (0:nelem, ncell)).  work: nslot*ncell + ncell doubles.
int launch_opacity_bwd(slg_ctx* ctx, const slg_gas* gas, const double* gcap, const double* gsig, double* gT,
                       double* goc, double* gnelec, double* gnatom, double* gfr, double* sig_work, double* work) {
  slg_opacity_flags fl{0, 0, 0, 0, 1, 0.0};
  OpacArgs A;
  int rc = opacity_prepare(ctx, gas, &fl, sig_work, A);
  if (rc) return rc;
  const int nc = ctx->nx, nslot = A.nelem * A.nst;
  double* ggrnd = work;
  double* ghlp = work + (size_t)nslot * nc;
  cudaStream_t st = ctx->stream;
  cudaMemsetAsync(ggrnd, 0, sizeof(double) * ((size_t)nslot * nc + nc), st);
  cudaMemsetAsync(goc, 0, sizeof(double) * (size_t)nslot * nc, st);
  cudaMemsetAsync(gfr, 0, sizeof(double) * (size_t)nc * (A.nelem + 1), st);
  OpacBwd B{gcap, gT, ggrnd, goc, ghlp, gfr};
  // the active slots, for the bound-free product
  int16_t* d_act = (int16_t*)scratch(ctx, 10, sizeof(int16_t) * (size_t)nslot);
  int* d_nact = (int*)scratch(ctx, 85, sizeof(int));
  if (!d_act || !d_nact) return SLG_ERR_OOM;
  ion_compact_kernel<<<1, 32, 0, st>>>(A.nelem, A.nst, ctx->d_ion_ni, A.active, d_act, d_nact);
  A.act_slot = d_act;
  A.pnact = d_nact;
  // two shells per lane where there are two warps of them (whole adjoint calls on
  // B200, one / two shells: 32 x 100 353 / 366 us, 64 x 100 354 / 365, 256 x 2000
  // 393 / 351, 4096 x 2000 3.70 / 3.12 ms)
  const int fs = nc <= OPAC_CT ? 1 : 2, gpb = groups_per_block(nc, A.ng, 8);
  const int tiles = (nc + fs * OPAC_CT - 1) / (fs * OPAC_CT), warps = tiles < kOpacWarps ? tiles : kOpacWarps;
  const dim3 grid((A.ng + gpb - 1) / gpb, (tiles + warps - 1) / warps);
  if (A.nobb) {  // no lines set
  } else if (fs == 2) {
    opacity_bwd_kernel<2><<<grid, warps * 32, 0, st>>>(A, B, ExpConst{}, gpb);
  } else {
    opacity_bwd_kernel<1><<<grid, warps * 32, 0, st>>>(A, B, ExpConst{}, gpb);
  }
  {
    // a block per shell, its groups split where that leaves less than four blocks an SM
    const int parts = (A.ng + 32 * kFfK - 1) / (32 * kFfK), fw = parts < kFfWarps ? parts : kFfWarps;
    const int want = (4 * ctx->num_sms + nc - 1) / nc, most = (parts + fw - 1) / fw;
    ff_bwd_kernel<<<dim3(nc, want < most ? want : most), fw * 32, 0, st>>>(A, B);
  }
  if (!A.nobf) {
    // about four blocks per SM over the slot tiles that a third of the slots fill
    // (the populated ones are known on the device only), of four tiles at least
    const int bx = (nc + BFB_T - 1) / BFB_T, by = (A.maxact + BFB_T - 1) / BFB_T;
    const int want = (4 * ctx->num_sms + bx * ((by + 2) / 3) - 1) / (bx * ((by + 2) / 3));
    const int most = (A.ng + 4 * BFB_T - 1) / (4 * BFB_T);
    const dim3 bgrid(bx, by, want < 1 ? 1 : want > most ? most : want);
    bf_bwd_kernel<<<bgrid, BFB_T * 8, 0, st>>>(A, B);
  }
  opac_cell_bwd_kernel<<<dim3((nc + 127) / 128, A.nelem), 128, 0, st>>>(nc, A.nelem, A.nst, ctx->d_ion_ni, gas->natom, gas->nelec,
                                                         gas->vol, gas->mass, gas->ginv, 0, ggrnd, ghlp, gsig, goc,
                                                         gnelec, gnatom);
  return cuda_check(ctx, cudaGetLastError(), "opacity adjoint launch");
}

// Sanity bitmask of physical_opacity.f:282-291 of the last build, on the device.
const int32_t* opacity_flags(slg_ctx* ctx) { return (const int32_t*)scratch(ctx, 3, sizeof(int) * 4); }

int launch_analytic_opacity(slg_ctx* ctx, const double* temp, const double* rho, int kind,
                            const double* c, double* gas_sig, float* gas_cap) {
  const int64_t nt = (int64_t)ctx->nx * ctx->ng;
  analytic_opacity_kernel<<<(unsigned)((nt + 255) / 256), 256, 0, ctx->stream>>>(
      ctx->nx, ctx->ng, ctx->d_wlinv, temp, rho, kind, c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7],
      gas_sig, gas_cap);
  return cuda_check(ctx, cudaGetLastError(), "analytic_opacity launch");
}

int launch_opacity_means(slg_ctx* ctx, const double* temp, const double* sig, const float* cap,
                         double* capgrey, double* capross) {
  launch_means(ctx, temp, sig, cap, capgrey, capross);
  return cuda_check(ctx, cudaGetLastError(), "opacity_means launch");
}

}  // namespace slg
