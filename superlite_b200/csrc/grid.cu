// grid.cu -- DDMC leakage opacities, emission probabilities and the per-cell
// tables of the transport kernels, for sm_100a.
//
// Reference: GRID/leakage_opacity11.f90:3-174, GRID/emission_probability.f90:3-67,
// GRID/emitgroup.f:3-54, TRANSPORT1/diffusion11.f90:95-152 (per-thread group
// cache) and the resolved-group sampling loops of diffusion11.f90:283-584.
//
// The reference rebuilds a per-thread cache (lump list, Planck weights) every
// time a DDMC particle enters a new cell and then scans up to ng groups per
// event to sample a resolved group.  Here every cell's cache and every scan's
// running partial sums are built once per call (build_cell_tables), in the
// reference's accumulation order, so a particle's linear scan "first position
// whose running sum exceeds r" becomes a binary search over the same
// sequence of partial sums (all terms are >= 0, so the sums are monotone).
#include <cuda_runtime.h>
#include <cfloat>
#include <type_traits>
#include "slg_device.cuh"
#include "slg_internal.h"

namespace slg {
namespace {

constexpr int GB = 256;  // block size of the per-cell kernels

__device__ inline double block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int w = GB / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + w];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// CT: opacity type, float (grd_cap) or double (the FP64 opacity of the
// differentiable path).
template <class CT>
struct LeakArgsT {
  int nx, ng;
  const double *xarr, *vol, *divv, *tempinv, *sig, *wlinv;
  const CT *cap, *capemit;
  double tauddmc, taulump;
  double* opaclump;
  const int4* cellmap;  // {shell, model shells, model first cell, model} per cell; null: one model
};
using LeakArgs = LeakArgsT<float>;

// Arguments seen from cell c (0-based over all models): per-cell arrays start
// at the cell's model, nx is the model's, *i the 1-based shell in the model.
template <class CT>
__device__ inline LeakArgsT<CT> leak_view(LeakArgsT<CT> A, int c, int* i) {
  *i = c + 1;
  if (A.cellmap) {
    const int4 m = A.cellmap[c];
    const int co = m.z;
    *i = m.x;
    A.nx = m.y;
    A.xarr += co + m.w;
    A.vol += co; A.divv += co; A.tempinv += co; A.sig += co;
    A.cap += (size_t)co * A.ng;
    if (A.capemit) A.capemit += (size_t)co * A.ng;
    A.opaclump += (size_t)11 * co;
  }
  return A;
}

// leakage_opacity11.f90:30-171.  One pass over the groups:
// one Planck weight per group and one division per face, the factors that the
// terms of a sum share (speclump, x^2 / vterm, divv / 3c) taken out of it.  The sums
// are fixed-shape tree reductions (the reference sums sequentially).  In four
// passes that each formed the weight anew, with eight block-wide reductions:
// 277 us at 28800 cells x 100 groups (now 39), 988 us at 4096 x 10000 in FP64 (640).
template <class CT, int FORM>
__global__ void __launch_bounds__(GB) leakage_kernel(const LeakArgsT<CT> A0, int nc) {
  constexpr int TPC = FORM == CELL_WARP ? 32 : GB;
  __shared__ double sh[6 * (GB / 32)];
  __shared__ double shv[GB / 32];
  __shared__ int shi[GB / 32];
  __shared__ double part[FORM == CELL_BLOCK_WARP_ORDER ? 6 * kWarpCellGroups : 1];
  const int cell = blockIdx.x * (GB / TPC) + threadIdx.x / TPC, t = threadIdx.x % TPC;
  if (cell >= nc) return;  // uniform over the cell's threads
  int i0;
  const LeakArgsT<CT> A = leak_view(A0, cell, &i0);
  const int i = i0;  // 1-based cell
  const int l = i, ng = A.ng;
  const double Xa = A.xarr[i - 1], Xb = A.xarr[i];
  const CT* capl = A.cap + (size_t)(l - 1) * ng;
  const double sigl = A.sig[l - 1];
  const double dist = Xb - Xa;
  const double tinv = A.tempinv[l - 1];
  const double hct = hck * tinv;
  const double divv = A.divv[l - 1];
  const bool in = i > 1, out = i < A.nx;  // a neighbour inside, outside
  const CT* cap1 = in ? capl - ng : capl;
  const CT* cap2 = out ? capl + ng : capl;
  const double sig1 = in ? A.sig[l - 2] : 0.0, sig2 = out ? A.sig[l] : 0.0;
  const double dx1 = in ? Xa - A.xarr[i - 2] : 0.0, dx2 = out ? A.xarr[i + 1] - Xb : 0.0;
  double bestv = 0.0;
  int besto = 0x7fffffff;
  // adds group ig to the sums: speclump, caplump, capemitlump, leakage left and right, doplump
  auto add = [&](int ig, double* a) {
    const double c = (double)capl[ig - 1];
    const double tau = (sigl + c) * dist;
    if (c * dist >= A.taulump && tau >= A.tauddmc) {
      const double sv = specintv_elem(hct, A.wlinv, ig - 1);
      a[0] = a[0] + sv;
      // caplump, capemitlump, igemitmax (first strict maximum over loop 1 then loop 2)
      const double h1 = sv * c;
      a[1] = a[1] + h1;
      if (h1 > bestv || (h1 == bestv && h1 > 0.0 && ig < besto)) { bestv = h1; besto = ig; }
      const double h2 = A.capemit ? sv * (double)A.capemit[(size_t)(l - 1) * ng + ig - 1] : 0.0;
      a[2] = a[2] + h2;
      if (h2 > bestv) { bestv = h2; besto = ng + ig; }
      // leakage: 1.5 * 4 / (3 tau + 6 dext) at a face to IMC, 2 / (tau + tau') inside
      const double tau1 = in ? ((double)cap1[ig - 1] + sig1) * dx1 : 0.0;
      const bool imc1 = !in || tau1 < A.tauddmc;
      a[3] = a[3] + sv * ((imc1 ? 6.0 : 2.0) / (imc1 ? 3.0 * tau + 6.0 * pc_dext : tau + tau1));
      const double tau2 = out ? ((double)cap2[ig - 1] + sig2) * dx2 : 0.0;
      const bool imc2 = !out || tau2 < A.tauddmc;
      a[4] = a[4] + sv * ((imc2 ? 6.0 : 2.0) / (imc2 ? 3.0 * tau + 6.0 * pc_dext : tau + tau2));
    }
    // doplump: a thick group whose next one (previous, for divv < 0) is not
    if (!(c * dist < A.taulump) && !(tau < A.tauddmc)) {
      if (divv >= 0.0) {
        if (ig < ng && !((double)capl[ig] * dist >= A.taulump)) a[5] = a[5] + dopspeccalc(tinv, A.wlinv, ig);
      } else {
        if (ig > 1 && !((double)capl[ig - 2] * dist >= A.taulump)) a[5] = a[5] - dopspeccalc(tinv, A.wlinv, ig - 1);
      }
    }
  };
  double a[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (FORM == CELL_BLOCK_WARP_ORDER) {
    for (int g = t; g < ng; g += TPC) {
      double e[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      add(g + 1, e);
#pragma unroll
      for (int k = 0; k < 6; ++k) part[k * kWarpCellGroups + g] = e[k];
    }
    cell_sum_of_block<6>(part, kWarpCellGroups, ng, a, sh);
  } else {
    for (int ig = t + 1; ig <= ng; ig += TPC) add(ig, a);
    cell_sum<TPC, 6>(a, sh);
  }
  auto better = [](double v2, int o2, double& v, int& o) {
    if (v2 > v || (v2 == v && o2 < o)) {
      v = v2;
      o = o2;
    }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    better(__shfl_xor_sync(0xffffffffu, bestv, o), __shfl_xor_sync(0xffffffffu, besto, o), bestv, besto);
  if (TPC > 32) {
    if ((threadIdx.x & 31) == 0) {
      shv[threadIdx.x >> 5] = bestv;
      shi[threadIdx.x >> 5] = besto;
    }
    __syncthreads();
    if (t == 0)
      for (int w = 1; w < GB / 32; ++w) better(shv[w], shi[w], bestv, besto);
  }
  if (t == 0) {
    const double speclump = a[0] > 0.0 ? 1.0 / a[0] : 0.0;
    const double vterm = 3.0 * A.vol[l - 1] / pc_pi4;
    int igemitmax = 0;
    if (bestv > 0.0) igemitmax = besto > ng ? besto - ng : besto;
    double* ol = A.opaclump + (size_t)11 * (l - 1);
    ol[0] = a[3] * speclump * (sq(Xa) / vterm);
    ol[1] = a[4] * speclump * (sq(Xb) / vterm);
    ol[2] = 0.0; ol[3] = 0.0; ol[4] = 0.0; ol[5] = 0.0;
    ol[6] = speclump;
    ol[7] = a[1];
    ol[8] = a[2];
    ol[9] = (double)igemitmax;
    ol[10] = a[5] * divv / (3.0 * pc_c);
  }
}

// emission_probability.f90:40-63: bin sums are sequential within a bin (one
// thread per bin) and the running sum over bins is sequential (one thread), as
// in the reference.  The terms are formed by all TPC threads of a cell first,
// bins_per_tile whole bins at a time, in shared memory (tile doubles per cell,
// then nep for the bin sums); with a thread per bin forming its own terms most
// of a block idled: 84 us at 28800 cells x 100 groups (now 24), 55 us at 1001 x 4003
// (35).
template <int TPC>
__global__ void __launch_bounds__(GB) emitprob_kernel(int nc, int ng, int nep, int nepg, int bins_per_tile,
                                                      const double* __restrict__ tempinv,
                                                      const float* __restrict__ cap,
                                                      const double* __restrict__ capgrey,
                                                      const double* __restrict__ wlinv,
                                                      double* __restrict__ emitprob) {
  extern __shared__ double s_dyn[];
  const int tile = bins_per_tile * nepg;
  double* const term = s_dyn + (size_t)(threadIdx.x / TPC) * (tile + nep);
  double* const binsum = term + tile;
  const int l = blockIdx.x * (GB / TPC) + threadIdx.x / TPC, t = threadIdx.x % TPC;
  if (l >= nc) return;  // uniform over the cell's threads
  double* ep = emitprob + (size_t)nep * l;
  if (ng == 1) {
    if (t == 0) ep[0] = capgrey[l];
    return;
  }
  auto sync = [] {
    if (TPC == 32) __syncwarp();
    else __syncthreads();
  };
  const double hct = hck * tempinv[l];
  const float* capl = cap + (size_t)l * ng;
  for (int b0 = 0; b0 < nep - 1; b0 += bins_per_tile) {
    const int g0 = b0 * nepg, n = min(min(b0 + bins_per_tile, nep - 1) * nepg, ng) - g0;
    sync();
    for (int k = t; k < n; k += TPC) term[k] = specintv_elem(hct, wlinv, g0 + k) * (double)capl[g0 + k];
    sync();
    for (int b = b0 + t; b < min(b0 + bins_per_tile, nep - 1); b += TPC) {
      double s = 0.0;
      const int top = min((b + 1) * nepg, ng) - g0;
      for (int k = b * nepg - g0; k < top; ++k) s = s + term[k];
      binsum[b] = s;
    }
  }
  sync();
  if (t == 0) {
    double help = 0.0;
    for (int iep = 1; iep <= nep - 1; ++iep) {
      help = help + binsum[iep - 1];
      ep[iep - 1] = help;
    }
    ep[nep - 1] = capgrey[l];
  }
}

// specintv_elem and its d/dT, from one exp, and the d/dT of dopspeccalc
// (groupmod.f:123-143, :189-198) at temperature T: x = hc/(lambda k T) scales as
// 1/T; zero derivative where x is clamped.
__device__ inline double spec_dT(double hct, double Tinv, const double* __restrict__ wlinv, int g0, double& dT) {
  const double x1 = hct * wlinv[g0], x2 = hct * wlinv[g0 + 1];
  const double xm = 0.5 * (x2 + x1), ax = fabs(x2 - x1);
  double fp, dfp = 0.0;
  if (xm >= 300.0) {
    fp = fplanck(xm);
  } else {
    const double ex = exp(xm), dinv = 1.0 / (ex - 1.0);
    fp = cube(xm) * dinv;
    dfp = (3.0 * sq(xm) - fp * ex) * dinv;
  }
  dT = -(ftpi4 * ax * (fp + xm * dfp)) * Tinv;
  return ftpi4 * ax * fp;
}
__device__ inline double ddop_dT(double tinv, const double* __restrict__ wlinv, int ig) {
  const double x = hck * tinv * wlinv[ig];
  if (x >= 300.0) return 0.0;
  const double ex = exp(x);
  return -dopspeccalc(tinv, wlinv, ig) * tinv * (4.0 - x * ex / (ex - 1.0));
}

// Adjoint of leakage_kernel<double>, a block per cell: adds to gcap, gsig and gT.
// Bound by FP64 issue and by the three reductions in memory per lumped group
// (its own and its neighbours' opacity): one exp and three divisions per group;
// with seven divisions 757 us at 4096 x 10000 (now 673).
__global__ void __launch_bounds__(GB, 4) leakage_bwd_kernel(const LeakArgsT<double> A0, const double* __restrict__ gol,
                                                         double* __restrict__ gcap, double* __restrict__ gsig,
                                                         double* __restrict__ gT) {
  __shared__ double sh[GB];
  const int c = blockIdx.x;  // cell over all models, 0-based
  int i0;
  const LeakArgsT<double> A = leak_view(A0, c, &i0);
  const int i = i0, ng = A.ng;
  const double* capl = A.cap + (size_t)(i - 1) * ng;
  const double sigl = A.sig[i - 1];
  const double dist = A.xarr[i] - A.xarr[i - 1];
  const double tinv = A.tempinv[i - 1];
  const double hct = hck * tinv;
  const double divv = A.divv[i - 1];
  const double* ol = A.opaclump + (size_t)11 * (i - 1);
  const double* u = gol + (size_t)11 * c;
  const double speclump = ol[6], ol1 = ol[0], ol2 = ol[1];
  const double u1 = u[0], u2 = u[1], u7 = u[6], u8 = u[7], u11 = u[10];
  const double vterm = 3.0 * A.vol[i - 1] / pc_pi4;
  const double fa = sq(A.xarr[i - 1]) / vterm, fb = sq(A.xarr[i]) / vterm;
  const bool in = i > 1, out = i < A.nx;  // a neighbour inside, outside
  const double sig1 = in ? A.sig[i - 2] : 0.0, sig2 = out ? A.sig[i] : 0.0;
  const double dx1 = in ? A.xarr[i - 1] - A.xarr[i - 2] : 0.0, dx2 = out ? A.xarr[i + 1] - A.xarr[i] : 0.0;
  double gs = 0.0, gt = 0.0, gsl = 0.0, gsr = 0.0;  // gsl, gsr: the neighbours' sigma, reduced once per block
  for (int ig = threadIdx.x + 1; ig <= ng; ig += GB) {
    const double cg = capl[ig - 1];
    if (!(cg * dist >= A.taulump && (sigl + cg) * dist >= A.tauddmc)) continue;
    double dsv;
    const double sv = spec_dT(hct, tinv, A.wlinv, ig - 1, dsv);
    // left leakage term a and d a / d(opacity sum) of this cell (da) and the left one (dal):
    // 6 fa / (3 tau + 6 dext) at a face to IMC, 2 fa / (tau + tau') inside
    const double tau = (cg + sigl) * dist;
    const double taul = in ? (A.cap[(size_t)(i - 2) * ng + ig - 1] + sig1) * dx1 : 0.0;
    const bool lint = in && taul >= A.tauddmc;
    const double qa = 1.0 / (lint ? tau + taul : 3.0 * tau + 6.0 * pc_dext);
    const double a = (lint ? 2.0 : 6.0) * fa * qa;
    const double ka = -a * qa, da = ka * (lint ? dist : 3.0 * dist), dal = ka * dx1;
    const double taur = out ? (A.cap[(size_t)i * ng + ig - 1] + sig2) * dx2 : 0.0;
    const bool rint = out && taur >= A.tauddmc;
    const double qb = 1.0 / (rint ? tau + taur : 3.0 * tau + 6.0 * pc_dext);
    const double b = (rint ? 2.0 : 6.0) * fb * qb;
    const double kb = -b * qb, db = kb * (rint ? dist : 3.0 * dist), dbr = kb * dx2;
    // ol1 = sum w_g a_g with w_g = sv_g speclump and speclump = 1/sum sv: d ol1/d sv_g = speclump (a_g - ol1)
    const double ua = u1 * sv * speclump, ub = u2 * sv * speclump;
    const double us = u1 * speclump * (a - ol1) + u2 * speclump * (b - ol2) - u7 * speclump * speclump + u8 * cg;
    gt += us * dsv;
    atomicAdd(&gcap[(size_t)c * ng + ig - 1], u8 * sv + ua * da + ub * db);
    gs += ua * da + ub * db;
    if (lint) {
      atomicAdd(&gcap[(size_t)(c - 1) * ng + ig - 1], ua * dal);
      gsl += ua * dal;
    }
    if (rint) {
      atomicAdd(&gcap[(size_t)(c + 1) * ng + ig - 1], ub * dbr);
      gsr += ub * dbr;
    }
  }
  if (u11 != 0.0) {
    if (divv >= 0.0) {
      for (int ig = threadIdx.x + 1; ig <= ng - 1; ig += GB) {
        if (capl[ig - 1] * dist < A.taulump || capl[ig] * dist >= A.taulump) continue;
        if ((sigl + capl[ig - 1]) * dist < A.tauddmc) continue;
        gt += u11 * ddop_dT(tinv, A.wlinv, ig) * divv / (3.0 * pc_c);
      }
    } else {
      for (int ig = threadIdx.x + 2; ig <= ng; ig += GB) {
        if (capl[ig - 1] * dist < A.taulump || capl[ig - 2] * dist >= A.taulump) continue;
        if ((sigl + capl[ig - 1]) * dist < A.tauddmc) continue;
        gt -= u11 * ddop_dT(tinv, A.wlinv, ig - 1) * divv / (3.0 * pc_c);
      }
    }
  }
  gs = block_sum(gs, sh);
  gt = block_sum(gt, sh);
  gsl = block_sum(gsl, sh);
  gsr = block_sum(gsr, sh);
  if (threadIdx.x == 0) {
    atomicAdd(&gsig[c], gs);
    gT[c] += gt;
    if (gsl != 0.0) atomicAdd(&gsig[c - 1], gsl);
    if (gsr != 0.0) atomicAdd(&gsig[c + 1], gsr);
  }
}

struct TabArgs {
  int nx, ng, nep, nepg;
  const double *xarr, *vxarr, *divv, *wlinv, *tempinv, *sig, *capgrey, *opaclump, *emitprob;
  const float* cap;
  double tauddmc, taulump;
  CellTables T;
  const int4* cellmap = nullptr;  // as LeakArgs::cellmap
  int fp64 = 1;                   // build what only the FP64 loop reads
};

// Arguments seen from cell c (see leak_view); *ic is the 1-based shell.
__device__ inline TabArgs tab_view(TabArgs A, int c, int* ic) {
  *ic = c + 1;
  if (A.cellmap) {
    const int4 m = A.cellmap[c];
    const int co = m.z;
    const size_t cg = (size_t)co * A.ng;
    *ic = m.x;
    A.nx = m.y;
    A.xarr += co + m.w; A.vxarr += co + m.w;
    A.divv += co; A.tempinv += co; A.sig += co; A.capgrey += co;
    A.opaclump += (size_t)11 * co;
    A.emitprob += (size_t)A.nep * co;
    A.cap += cg;
    A.T.specarr += cg; A.T.glumps += cg;
    if (A.fp64) {
      A.T.cdf_dop += cg; A.T.cdf_left += cg; A.T.cdf_right += cg; A.T.cdf_scat += cg;
      A.T.emitcum += cg;
    } else {
      A.T.sum_dop += cg; A.T.sum_left += cg; A.T.sum_right += cg; A.T.sum_scat += cg;
    }
    if (A.T.guide) A.T.guide += (size_t)co * 4 * (A.T.guide_m + 1);
    if (A.T.fine) A.T.fine += (size_t)co * kFineTables * A.T.fine_m;
    A.T.nlump += co;
    A.T.scal += (size_t)SCAL_N * co;
  }
  return A;
}

// CdfEntry::info of group ig of cell l (1-based; c: its opacity, dist: its width).
__device__ inline int group_info(const TabArgs& A, int l, double dist, int ig, double c) {
  if ((A.sig[l - 1] + c) * dist < A.tauddmc) return ig | kInfoImc;
  const bool lumped = c * dist >= A.taulump && A.opaclump[(size_t)11 * (l - 1) + 6] != 0.0;
  return lumped ? ig | kInfoLumped : ig;
}

// An entry of a running sum in either loop's form.
__device__ inline double& sum_of(CdfEntry& e) { return e.sum; }
__device__ inline double& sum_of(double& e) { return e; }
__device__ inline CdfEntry make_entry(const CdfEntry*, double sum, int info) { return CdfEntry{sum, info, 0}; }
__device__ inline double make_entry(const double*, double sum, int) { return sum; }

// In-place running sum in index order by a warp: a chain of dependent FP64
// additions by its first lane, over tiles that the warp loads and stores together
// (tile: kSumTile doubles of shared memory; the next tile's terms are under way
// meanwhile).  With a load and a store in memory for each entry the requests of all
// blocks' four chains took 600 of the kernel's 1060 us at 1024 cells x 4000 groups; as
// an addition of every lane, with the terms exchanged by shuffles, 230.
constexpr int kSumTile = 128;
template <class E>
__device__ inline void running_sum(E* __restrict__ a, int n, double* tile) {
  constexpr int PER = kSumTile / 32, N = 8;
  const int lane = threadIdx.x & 31;
  double v[PER], s = 0.0;
#pragma unroll
  for (int k = 0; k < PER; ++k) v[k] = 32 * k + lane < n ? sum_of(a[32 * k + lane]) : 0.0;
  for (int q = 0; q < n; q += kSumTile) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      tile[32 * k + lane] = v[k];
      const int next = q + kSumTile + 32 * k + lane;
      v[k] = next < n ? sum_of(a[next]) : 0.0;
    }
    __syncwarp();
    if (lane == 0) {
      const int m = min(n - q, kSumTile);
      for (int k = 0; k < m; k += N) {
        double2 t[N / 2];
#pragma unroll
        for (int j = 0; j < N / 2; ++j) t[j] = reinterpret_cast<double2*>(tile + k)[j];
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
          t[j].x = s + t[j].x;
          t[j].y = t[j].x + t[j].y;
          s = t[j].y;
          reinterpret_cast<double2*>(tile + k)[j] = t[j];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (q + 32 * k + lane < n) sum_of(a[q + 32 * k + lane]) = tile[32 * k + lane];
    __syncwarp();
  }
}

// 1 / (sum of the branch rates) and the branch limits {P(Doppler), P(Doppler) +
// P(left leak)} (diffusion11.f90:232-278).
__device__ inline double2 ddmc_rates(double o1, double o2, double emitlump, double caplump, double doplump,
                                     double* denom) {
  double d = (o1 + o2) + (1.0 - emitlump) * caplump + doplump;
  d = 1.0 / d;
  *denom = d;
  const double pdop = doplump * d;
  return make_double2(pdop, pdop + o1 * d);
}

// number of leading entries of a (n, non-decreasing) not above v
__device__ inline int count_le(const double* __restrict__ a, int n, double v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] <= v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The ranges {first, last} of one table of CellTables::fine, by the whole block:
// range k holds the numbers of entries that limits k and k + 1 do not lie below.
// first_limit(i): the first limit that does not lie below entry i (fm + 1: none of the
// fm + 1), non-decreasing in i, so that a limit's number is the largest i + 1 of the
// entries whose first limit is not above it: a maximum per limit, then a running one.
// lim: fm + 1 ints of shared memory, wmax: GB / 32.  (A search of the table for every
// limit took 290 of the kernel's 1060 us at 1024 cells x 4000 groups, this 107.)
template <class First>
__device__ inline void fine_ranges(short2* __restrict__ fd, int fm, int n, int* lim, int* wmax, First first_limit) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (int k = t; k <= fm; k += GB) lim[k] = 0;
  __syncthreads();
  for (int i = t; i < n; i += GB) {
    const int k = first_limit(i);
    if (k <= fm) atomicMax(&lim[k], i + 1);
  }
  __syncthreads();
  const int per = fm / GB + 1, k0 = min(t * per, fm + 1), k1 = min(k0 + per, fm + 1);
  int m = 0;
  for (int k = k0; k < k1; ++k) m = max(m, lim[k]);
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, m, o);
    if (lane >= o) m = max(m, v);
  }
  if (lane == 31) wmax[wid] = m;
  m = __shfl_up_sync(0xffffffffu, m, 1);
  if (lane == 0) m = 0;
  __syncthreads();
  for (int w = 0; w < wid; ++w) m = max(m, wmax[w]);
  for (int k = k0; k < k1; ++k) {
    m = max(m, lim[k]);
    lim[k] = m;
  }
  __syncthreads();
  for (int k = t; k < fm; k += GB) fd[k] = make_short2((short)lim[k], (short)lim[k + 1]);
  __syncthreads();
}

// TrnCell record of shell ix, from its scalars (CellTables::scal, nlump).
__device__ inline TrnCell cell_record(const TabArgs& A, int ix) {
  const double* X = A.xarr;
  const double* sc = A.T.scal + (size_t)SCAL_N * (ix - 1);
  TrnCell r;
  r.xa = X[ix - 1];
  r.xb = X[ix];
  r.vxa = A.vxarr[ix - 1];
  r.vxb = A.vxarr[ix];
  r.dist = r.xb - r.xa;
  r.sig = A.sig[ix - 1];
  r.divv = A.divv[ix - 1];
  r.capgrey = A.capgrey[ix - 1];
  r.x0 = X[0];
  r.far = sc[SCAL_FAR];
  r.dvdr = sc[SCAL_DVDR];
  r.vhelp = r.vxa - r.dvdr * r.xa;
  r.dopc = 3.0 * pc_c / r.divv;
  r.sigl = ix > 1 ? A.sig[ix - 2] : 0.0;
  r.dxl = ix > 1 ? X[ix - 1] - X[ix - 2] : 0.0;
  r.divvl = ix > 1 ? A.divv[ix - 2] : 0.0;
  r.sigr = ix < A.nx ? A.sig[ix] : 0.0;
  r.dxr = ix < A.nx ? X[ix + 1] - X[ix] : 0.0;
  r.divvr = ix < A.nx ? A.divv[ix] : 0.0;
  r.xa3 = cube(r.xa);
  r.xb3 = cube(r.xb);
  r.nlump = A.T.nlump[ix - 1];
  r.pad = 0;
  const double* OL = A.opaclump + (size_t)11 * (ix - 1);
  const double2 lo = ddmc_rates(OL[0], OL[1], sc[SCAL_EMITLUMP], sc[SCAL_CAPLUMP], sc[SCAL_DOPLUMP], &r.denom);
  r.pdop = lo.x;
  r.pleft = lo.y;
  r.pleak = lo.x + (OL[0] * r.denom + OL[1] * r.denom);
  return r;
}

// Per-cell transport tables (see CellTables).  Phase A computes every term in
// parallel; phase B forms the running sums sequentially, a warp per table,
// in the order of the reference's loops; phase C the guides.  Bound by phase A's
// exponentials and divisions and by the chains of phase B.  A whole FP64 launch
// without a particle on B200 (with ddmc_rate_kernel; what a launch pays before its
// events): 256 cells x 2000 groups 225 -> 130 us, 1024 x 4000 1190 -> 529, 4000 x 100 235
// -> 154, against 116, 420 and 123 without tables for the events, each of which
// takes a microsecond or two less with them: longest histories of some hundred
// events pay for the tables.  Four blocks per SM: three / four / five 592 / 529 / 545 us
// at 1024 x 4000.
template <bool FP64>
__global__ void __launch_bounds__(GB, 4) cell_tables_kernel(const TabArgs A0) {
  __shared__ int warp_l[GB / 32], warp_u[GB / 32];
  __shared__ int base_l, base_u;
  __shared__ __align__(16) double tile[4][kSumTile];
  __shared__ int lim[kFineMax + 1];
  int ic0;
  const TabArgs A = tab_view(A0, blockIdx.x, &ic0);
  const int ic = ic0, ix = ic;
  const int ng = A.ng;
  const size_t off = (size_t)(ic - 1) * ng;
  const float* capc = A.cap + off;
  const double dist = A.xarr[ix] - A.xarr[ix - 1];
  const double sigc = A.sig[ic - 1];
  const double tinv = A.tempinv[ic - 1];
  const double hct = hck * tinv;
  const double* OL = A.opaclump + (size_t)11 * (ic - 1);
  const double speclump = OL[6];
  double* specarr = A.T.specarr + off;
  int16_t* glumps = A.T.glumps + off;
  // specarr and the lump ordering (diffusion11.f90:103-124)
  if (threadIdx.x == 0) { base_l = 0; base_u = 0; }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c0 = 0; c0 < ng; c0 += GB) {
    const int ig = c0 + threadIdx.x + 1;
    bool lump = false;
    if (ig <= ng) {
      specarr[ig - 1] = specintv_elem(hct, A.wlinv, ig - 1);
      const double c = (double)capc[ig - 1];
      lump = speclump != 0.0 && c * dist >= A.taulump && (sigc + c) * dist >= A.tauddmc;
    }
    const unsigned bl = __ballot_sync(0xffffffffu, ig <= ng && lump);
    const unsigned bu = __ballot_sync(0xffffffffu, ig <= ng && !lump);
    if (lane == 0) { warp_l[wid] = __popc(bl); warp_u[wid] = __popc(bu); }
    __syncthreads();
    int pl = base_l, pu = base_u;
    for (int w = 0; w < wid; ++w) { pl += warp_l[w]; pu += warp_u[w]; }
    const unsigned below = (1u << lane) - 1u;
    pl += __popc(bl & below);
    pu += __popc(bu & below);
    if (ig <= ng) {
      if (lump) glumps[pl] = (int16_t)ig;              // glumps(pl+1)
      else if (speclump != 0.0) glumps[ng - 1 - pu] = (int16_t)ig;  // glumps(ng-pu)
      else glumps[ig - 1] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 0; w < GB / 32; ++w) { base_l += warp_l[w]; base_u += warp_u[w]; }
    }
    __syncthreads();
  }
  const int nlump = base_l;
  // scalars (diffusion11.f90:98-150)
  const double cgi0 = 1.0 / A.capgrey[ic - 1];
  const double capgreyinv = cgi0 > 0.0 ? cgi0 : 0.0;
  double emitlump, caplump, doplump;
  if (nlump == ng) {
    emitlump = 1.0;
    caplump = A.capgrey[ic - 1];
    doplump = 0.0;
  } else {
    caplump = OL[7] * speclump;
    emitlump = OL[7] * capgreyinv;
    emitlump = emitlump < 1.0 ? emitlump : 1.0;
    doplump = OL[10] * speclump;
  }
  const double X0 = A.xarr[ix - 1], X1 = A.xarr[ix];
  const double dx3 = cube(X1) - cube(X0);
  if (threadIdx.x == 0) {
    A.T.nlump[ic - 1] = nlump;
    double* sc = A.T.scal + (size_t)SCAL_N * (ic - 1);
    sc[SCAL_EMITLUMP] = emitlump;
    sc[SCAL_CAPLUMP] = caplump;
    sc[SCAL_DOPLUMP] = doplump;
    sc[SCAL_CAPGREYINV] = capgreyinv;
    sc[SCAL_SPECLUMP] = speclump;
    sc[SCAL_FAR] = 2.0 * fabs(sqrt(sq(X1) - sq(X0)));
    sc[SCAL_DX3] = dx3;
    sc[SCAL_DVDR] = (A.vxarr[ix] - A.vxarr[ix - 1]) / dist;
    if (FP64) A0.T.cell[blockIdx.x] = cell_record(A, ix);
  }
  __syncthreads();  // glumps and specarr visible to the block
  const double divv = A.divv[ix - 1];
  using E = typename std::conditional<FP64, CdfEntry, double>::type;
  E *cdop, *cleft, *cright, *cscat;
  if constexpr (FP64) {
    cdop = A.T.cdf_dop + off; cleft = A.T.cdf_left + off; cright = A.T.cdf_right + off; cscat = A.T.cdf_scat + off;
  } else {
    cdop = A.T.sum_dop + off; cleft = A.T.sum_left + off; cright = A.T.sum_right + off; cscat = A.T.sum_scat + off;
  }
  double* ecum = A.T.emitcum + off;
  // ---- phase A: terms
  if (nlump > 0) {
    const double hdop = 1.0 / doplump;
    const double hl = 1.0 / OL[0], hr = 1.0 / OL[1];
    const double denom2 = 1.0 / (1.0 - emitlump);
    for (int q = threadIdx.x + 1; q <= ng; q += GB) {
      // Doppler (diffusion11.f90:290-314): position q in loop order
      if (q <= nlump) {
        double t = 0.0;
        int from, to;  // the resolved group and the one it shifts to
        if (divv >= 0.0) {
          const int iiig = glumps[q - 1];
          from = iiig;
          to = min(iiig + 1, ng);
          if (!(iiig == ng) && !((double)capc[iiig] * dist >= A.taulump)) {
            const double res = dopspeccalc(tinv, A.wlinv, iiig) * divv / (3.0 * pc_c);
            t = res * speclump * hdop;
          }
        } else {
          const int iig = nlump + 1 - q;
          const int iiig = glumps[iig - 1];
          from = iiig;
          to = max(iiig - 1, 1);
          if (!(iiig == 1) && !((double)capc[iiig - 2] * dist >= A.taulump)) {
            const double res = dopspeccalc(tinv, A.wlinv, iiig - 1) * divv / (3.0 * pc_c);
            t = -(res * speclump * hdop);
          }
        }
        cdop[q - 1] = make_entry(cdop, t, from | (group_info(A, ic, dist, to, (double)capc[to - 1]) & ~0xffff));
        // left leak (:378-397)
        const int iiig = glumps[q - 1];
        const double specig = specarr[iiig - 1];
        const double capi = (double)capc[iiig - 1];
        if (ix > 1) {
          const int l = ix - 1;
          const double capl = (double)A.cap[(size_t)(l - 1) * ng + iiig - 1];
          const double dxl = A.xarr[ix - 1] - A.xarr[ix - 2];
          double res;
          if ((capl + A.sig[l - 1]) * dxl < A.tauddmc) {
            const double mfphelp = (capi + sigc) * dist;
            const double ppl = 4.0 / (3.0 * mfphelp + 6.0 * pc_dext);
            res = 1.5 * ppl * sq(X0) / dx3;
          } else {
            const double mfphelp = (sigc + capi) * dist + (A.sig[l - 1] + capl) * dxl;
            res = 2.0 * sq(X0) / (mfphelp * dx3);
          }
          cleft[q - 1] = make_entry(cleft, specig * res * speclump * hl, group_info(A, l, dxl, iiig, capl));
        }
        // right leak: boundary (:450-460) or interior (:492-511)
        double res;
        int info = iiig;
        if (ix == A.nx) {
          const double mfphelp = (capi + sigc) * dist;
          const double ppr = 4.0 / (3.0 * mfphelp + 6.0 * pc_dext);
          res = 1.5 * ppr * sq(X1) / dx3;
        } else {
          const int l = ix + 1;
          const double capl = (double)A.cap[(size_t)(l - 1) * ng + iiig - 1];
          const double dxr = A.xarr[ix + 1] - A.xarr[ix];
          info = group_info(A, l, dxr, iiig, capl);
          if ((capl + A.sig[l - 1]) * dxr < A.tauddmc) {
            const double mfphelp = (capi + sigc) * dist;
            const double ppr = 4.0 / (3.0 * mfphelp + 6.0 * pc_dext);
            res = 1.5 * ppr * sq(X1) / dx3;
          } else {
            const double mfphelp = (sigc + capi) * dist + (A.sig[l - 1] + capl) * dxr;
            res = 2.0 * sq(X1) / (mfphelp * dx3);
          }
        }
        cright[q - 1] = make_entry(cright, specig * res * speclump * hr, info);
      }
      // effective scattering over unlumped groups (:571-584), loop order q
      if (q <= ng - nlump) {
        const int iig = ng + 1 - q;
        const int iiig = glumps[iig - 1];
        const double help = specarr[iiig - 1] * (double)capc[iiig - 1] * capgreyinv;
        cscat[q - 1] = make_entry(cscat, help * denom2, group_info(A, ic, dist, iiig, (double)capc[iiig - 1]));
      }
    }
  }
  // emitgroup's thresholds (emitgroup.f:303-320), one thread per emission bin.
  // The reference takes the bin iep = number of ep(1:nep-1) not above r1 and in
  // it the first group whose running sum from ep(iep) exceeds r1, else the
  // bin's last.  Flattened over the bins, entry g-1 is the r1 from which the
  // answer passes group g: the running sum inside a bin, kept from passing the
  // next bin's start (which rounding could otherwise do), and that start at
  // the bin's last group.  The entries are non-decreasing, so the answer is
  // one plus the number of entries not above r1.
  if (FP64) {
    const double* ep = A.emitprob + (size_t)A.nep * (ic - 1);
    const int last = emit_last_group(A.nep, A.nepg, ng);
    for (int iep = threadIdx.x; iep < A.nep; iep += GB) {
      const int ig0 = iep * A.nepg + 1;
      const int igp1 = min(ig0 + A.nepg - 1, last);
      double prob = iep == 0 ? 0.0 : ep[iep - 1];
      const bool end = iep == A.nep - 1;
      const double next = end ? DBL_MAX : ep[iep];
      for (int g = ig0; g <= igp1 - 1; ++g) {
        prob = prob + specarr[g - 1] * (double)capc[g - 1];
        ecum[g - 1] = !end && prob > next ? next : prob;
      }
      if (igp1 >= ig0 && igp1 < last) ecum[igp1 - 1] = next;
    }
  }
  __syncthreads();
  // ---- phase B: running sums
  if (nlump > 0) {
    if (wid == 0) running_sum(cdop, nlump, tile[0]);
    else if (wid == 1 && ix > 1) running_sum(cleft, nlump, tile[1]);
    else if (wid == 2) running_sum(cright, nlump, tile[2]);
    else if (wid == 3) running_sum(cscat, ng - nlump, tile[3]);
  }
  // ---- phase C: guide tables: the mixed loop's (CellTables::guide) or the FP64 loop's
  __syncthreads();
  if constexpr (!FP64) {
    if (!A.T.guide || nlump == 0) return;
    const int gm = A.T.guide_m;
    int16_t* gd = A.T.guide + (size_t)(ic - 1) * 4 * (gm + 1);
    for (int t = 0; t < 4; ++t) {
      const E* a = t == 0 ? cdop : (t == 1 ? cleft : (t == 2 ? cright : cscat));
      const int n = t == 3 ? ng - nlump : nlump;
      for (int k = threadIdx.x; k <= gm; k += blockDim.x)  // no left leak from the first shell
        gd[t * (gm + 1) + k] = (int16_t)count_le(a, t == 1 && ix == 1 ? 0 : n, (double)k / (double)gm);
    }
  }
  if constexpr (FP64) {
    if (!A.T.fine) return;
    const int fm = A.T.fine_m;
    short2* fd = A.T.fine + (size_t)(ic - 1) * kFineTables * fm;
    if (nlump > 0) {
      for (int t = 0; t < 4; ++t) {
        const CdfEntry* a = t == 0 ? cdop : (t == 1 ? cleft : (t == 2 ? cright : cscat));
        const int n = t == 1 && ix == 1 ? 0 : (t == 3 ? ng - nlump : nlump);  // no left leak from the first shell
        // limit k is k / fm (fm is a power of two: the products are exact)
        fine_ranges(fd + (size_t)t * fm, fm, n, lim, warp_l, [&](int i) {
          const double x = a[i].sum * (double)fm;
          return x <= (double)fm ? max((int)ceil(x), 0) : fm + 1;
        });
      }
    }
    // the emission thresholds: limit k is (k / fm) capgrey, rounded as a draw's
    // product by capgrey is
    const int n = emit_last_group(A.nep, A.nepg, ng) - 1;
    const double cg = A.capgrey[ic - 1];
    const int one = emit_only_group(A.nep, A.nepg, ng, cg != cg);
    if (one) {
      for (int k = threadIdx.x; k < fm; k += GB) fd[4 * fm + k] = make_short2((short)(one - 1), (short)(one - 1));
    } else {
      const double scale = (double)fm / cg;
      fine_ranges(fd + (size_t)4 * fm, fm, n, lim, warp_l, [&](int i) {
        const double e = ecum[i], x = e * scale;
        int k = x <= (double)fm ? max((int)x, 0) : (x != x ? 0 : fm + 1);  // near the limit: then to it
        while (k > 0 && !(e > ((double)(k - 1) / (double)fm) * cg)) --k;
        while (k <= fm && e > ((double)k / (double)fm) * cg) ++k;
        return k;
      });
    }
  }
}

// CellTables::rates, one thread per (cell, group): the branch rates that
// diffusion11.f90:154-278 forms for every event, once per entry (two exp and
// eight divisions), with the expressions in the reference's order.
__global__ void __launch_bounds__(256) ddmc_rate_kernel(const TabArgs A0, int nc, double2* __restrict__ out) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int ng = A0.ng;
  if (k >= (size_t)nc * ng) return;
  const int c = (int)(k / ng), ig = (int)(k - (size_t)c * ng) + 1;
  int ix;
  const TabArgs A = tab_view(A0, c, &ix);
  const double* X = A.xarr;
  const float* cap = A.cap + (size_t)(ix - 1) * ng + (ig - 1);
  const double Xa = X[ix - 1], Xb = X[ix], dist = Xb - Xa;
  const double sigc = A.sig[ix - 1], capc = (double)cap[0];
  double2 lo, hi = make_double2(0.0, 0.0);
  if ((sigc + capc) * dist < A.tauddmc) {
    lo = make_double2(__hiloint2double(kRateImcHi, 0), 0.0);
  } else if (capc * dist >= A.taulump && A.T.nlump[ix - 1] > 0) {
    lo = make_double2(__hiloint2double(kRateLumpedHi, 0), 0.0);
  } else {
    const double* sc = A.T.scal + (size_t)SCAL_N * (ix - 1);
    const double tinv = A.tempinv[ix - 1], divv = A.divv[ix - 1], dx3 = sc[SCAL_DX3];
    const double emitlump = specint0(tinv, A.wlinv, ig) * sc[SCAL_CAPGREYINV] * capc;
    const double spec_ig = A.T.specarr[(size_t)(ix - 1) * ng + ig - 1];
    double doplump;
    if (ig != ng && divv >= 0.0) {
      doplump = dopspeccalc(tinv, A.wlinv, ig) * divv / (spec_ig * 3.0 * pc_c);
    } else if (ig != 1 && divv < 0.0) {
      doplump = -1.0 * dopspeccalc(tinv, A.wlinv, ig - 1) * divv / (spec_ig * 3.0 * pc_c);
    } else {
      doplump = 0.0;
    }
    double o1 = 0.0, o2;
    if (ix > 1) {
      const double capl = (double)cap[-ng], sigl = A.sig[ix - 2];
      const double dxl = Xa - X[ix - 2];
      if ((capl + sigl) * dxl < A.tauddmc) {
        const double mfphelp = (capc + sigc) * dist;
        const double ppl = 4.0 / (3.0 * mfphelp + 6.0 * pc_dext);
        o1 = 1.5 * ppl * sq(Xa) / dx3;
      } else {
        const double mfphelp = (sigc + capc) * dist + (sigl + capl) * dxl;
        o1 = 2.0 * sq(Xa) / (mfphelp * dx3);
      }
    }
    bool lhelp = true;
    double capl = 0.0, sigl = 0.0, dxl = 0.0;
    if (ix != A.nx) {
      capl = (double)cap[ng];
      sigl = A.sig[ix];
      dxl = X[ix + 1] - Xb;
      lhelp = (capl + sigl) * dxl < A.tauddmc;
    }
    if (lhelp) {
      const double mfphelp = (capc + sigc) * dist;
      const double ppr = 4.0 / (3.0 * mfphelp + 6.0 * pc_dext);
      o2 = 1.5 * ppr * sq(Xb) / dx3;
    } else {
      const double mfphelp = (sigc + capc) * dist + (sigl + capl) * dxl;
      o2 = 2.0 * sq(Xb) / (mfphelp * dx3);
    }
    double denom;
    const double2 d = ddmc_rates(o1, o2, emitlump, capc, doplump, &denom);
    lo = make_double2(denom, d.x);
    hi = make_double2(d.y, d.x + (o1 * denom + o2 * denom));
  }
  out[2 * k] = lo;
  out[2 * k + 1] = hi;
}

}  // namespace

template <class CT>
static void launch_leakage_kernel(slg_ctx* ctx, const LeakArgsT<CT>& A) {
  const int nc = ctx->nx;
  switch (cell_form(nc, ctx->ng, ctx->num_sms)) {
    case CELL_WARP: leakage_kernel<CT, CELL_WARP><<<(nc + GB / 32 - 1) / (GB / 32), GB, 0, ctx->stream>>>(A, nc); break;
    case CELL_BLOCK_WARP_ORDER: leakage_kernel<CT, CELL_BLOCK_WARP_ORDER><<<nc, GB, 0, ctx->stream>>>(A, nc); break;
    default: leakage_kernel<CT, CELL_BLOCK><<<nc, GB, 0, ctx->stream>>>(A, nc);
  }
}

int launch_leakage(slg_ctx* ctx, const double* tempinv, const double* sig, const float* cap,
                   const float* capemit, double tauddmc, double taulump, double* opaclump) {
  LeakArgs A{ctx->nx, ctx->ng, ctx->d_xarr, ctx->d_vol, ctx->d_divv, tempinv, sig, ctx->d_wlinv,
             cap, capemit, tauddmc, taulump, opaclump, ctx->nmodel > 1 ? ctx->d_cellmap : nullptr};
  launch_leakage_kernel(ctx, A);
  return cuda_check(ctx, cudaGetLastError(), "leakage launch");
}

// leakage_opacity11 on the FP64 opacity (ng, ncell) of the differentiable path.
int launch_leakage64(slg_ctx* ctx, const double* tempinv, const double* sig, const double* cap, double tauddmc,
                     double taulump, double* opaclump) {
  LeakArgsT<double> A{ctx->nx, ctx->ng, ctx->d_xarr, ctx->d_vol, ctx->d_divv, tempinv, sig, ctx->d_wlinv,
                      cap, nullptr, tauddmc, taulump, opaclump, ctx->nmodel > 1 ? ctx->d_cellmap : nullptr};
  launch_leakage_kernel(ctx, A);
  return cuda_check(ctx, cudaGetLastError(), "leakage64 launch");
}

// Adjoint of leakage_kernel<double> for opaclump rows 1, 2 (leakage), 7
// (speclump), 8 (caplump) and 11 (doplump): gol (11, ncell) in; adds to gcap
// (ng, ncell) of the cell and its neighbours, gsig and gT.  The lumping masks
// are piecewise constant and contribute nothing.
int launch_leakage64_bwd(slg_ctx* ctx, const double* tempinv, const double* sig, const double* cap,
                         double tauddmc, double taulump, const double* opaclump, const double* gol, double* gcap,
                         double* gsig, double* gT) {
  LeakArgsT<double> A{ctx->nx, ctx->ng, ctx->d_xarr, ctx->d_vol, ctx->d_divv, tempinv, sig, ctx->d_wlinv,
                      cap, nullptr, tauddmc, taulump, const_cast<double*>(opaclump),
                      ctx->nmodel > 1 ? ctx->d_cellmap : nullptr};
  leakage_bwd_kernel<<<ctx->nx, GB, 0, ctx->stream>>>(A, gol, gcap, gsig, gT);
  return cuda_check(ctx, cudaGetLastError(), "leakage adjoint launch");
}

int launch_emitprob(slg_ctx* ctx, const double* tempinv, const float* cap, const double* capgrey,
                    double* emitprob) {
  // a tile: all bins of a cell where a warp takes it, else up to 4096 groups
  // (nepg is at most 181 for the largest group count)
  const int nc = ctx->nx, ng = ctx->ng, nep = ctx->nep, nepg = ctx->nepg;
  const bool warp = cell_form(nc, ng, ctx->num_sms) == CELL_WARP;  // (bins have one order in any form)
  const int cells = warp ? GB / 32 : 1, bins = warp ? nep : (4096 / nepg < nep ? 4096 / nepg : nep);
  const size_t shm = sizeof(double) * cells * ((size_t)bins * nepg + nep);  // at most 36 KB
  if (warp)
    emitprob_kernel<32><<<(nc + cells - 1) / cells, GB, shm, ctx->stream>>>(nc, ng, nep, nepg, bins, tempinv, cap,
                                                                           capgrey, ctx->d_wlinv, emitprob);
  else
    emitprob_kernel<GB><<<nc, GB, shm, ctx->stream>>>(nc, ng, nep, nepg, bins, tempinv, cap, capgrey, ctx->d_wlinv,
                                                     emitprob);
  return cuda_check(ctx, cudaGetLastError(), "emission_probability launch");
}

namespace {
void launch_tables(cudaStream_t st, int nx, const TabArgs& A) {
  if (!A.fp64) {
    cell_tables_kernel<false><<<nx, GB, 0, st>>>(A);
    return;
  }
  cell_tables_kernel<true><<<nx, GB, 0, st>>>(A);
  const size_t n = (size_t)nx * A.ng;
  ddmc_rate_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(A, nx, A.T.rates);
}
}  // namespace

int build_cell_tables(slg_ctx* ctx, const slg_transport_in* in) {
  const int nx = ctx->nx, ng = ctx->ng;
  const size_t n = (size_t)nx * ng;
  CellTables& T = ctx->tables;
  const bool fp64 = in->precision == 0;  // the mixed loop has its own rates and emission CDF
  if (T.nx != nx || T.ng != ng) {
    T.have_fp64 = T.have_mixed = false;
    T.specarr = (double*)scratch(ctx, 12, sizeof(double) * n);
    T.glumps = (int16_t*)scratch(ctx, 13, sizeof(int16_t) * n);
    T.nlump = (int32_t*)scratch(ctx, 19, sizeof(int32_t) * nx);
    T.scal = (double*)scratch(ctx, 20, sizeof(double) * SCAL_N * nx);
    T.guide_m = guide_size(ng);
    T.fine_m = fine_size(ng);
    if (!T.specarr || !T.glumps || !T.nlump || !T.scal) {
      T.nx = T.ng = 0;
      return SLG_ERR_OOM;
    }
  }
  // Each loop's tables have buffers of their own: a launch of one loop between the
  // replays of a graph that holds the other's moves nothing that the graph reads.
  // (Guide entries are int16 positions; SLG_MAX_GROUPS keeps to them.)
  bool ok = true;
  if (fp64 && !T.have_fp64) {
    T.cdf_dop = (CdfEntry*)scratch(ctx, 94, sizeof(CdfEntry) * n);
    T.cdf_left = (CdfEntry*)scratch(ctx, 95, sizeof(CdfEntry) * n);
    T.cdf_right = (CdfEntry*)scratch(ctx, 96, sizeof(CdfEntry) * n);
    T.cdf_scat = (CdfEntry*)scratch(ctx, 97, sizeof(CdfEntry) * n);
    T.emitcum = (double*)scratch(ctx, 18, sizeof(double) * n);
    T.rates = (double2*)scratch(ctx, 91, sizeof(double2) * 2 * n);
    T.cell = (TrnCell*)scratch(ctx, 92, sizeof(TrnCell) * (size_t)nx);
    T.fine = (short2*)scratch(ctx, 93, sizeof(short2) * kFineTables * T.fine_m * (size_t)nx);
    T.have_fp64 = ok = T.cdf_dop && T.cdf_left && T.cdf_right && T.cdf_scat && T.emitcum && T.rates && T.cell && T.fine;
  } else if (!fp64 && !T.have_mixed) {
    T.sum_dop = (double*)scratch(ctx, 14, sizeof(double) * n);
    T.sum_left = (double*)scratch(ctx, 15, sizeof(double) * n);
    T.sum_right = (double*)scratch(ctx, 16, sizeof(double) * n);
    T.sum_scat = (double*)scratch(ctx, 17, sizeof(double) * n);
    T.guide = (int16_t*)scratch(ctx, 72, sizeof(int16_t) * 4 * (T.guide_m + 1) * (size_t)nx);
    T.have_mixed = ok = T.sum_dop && T.sum_left && T.sum_right && T.sum_scat && T.guide;
  }
  if (!ok) {
    T.nx = T.ng = 0;
    return SLG_ERR_OOM;
  }
  T.nx = nx;
  T.ng = ng;
  TabArgs A;
  A.nx = nx; A.ng = ng; A.nep = ctx->nep; A.nepg = ctx->nepg;
  A.xarr = ctx->d_xarr; A.vxarr = ctx->d_vxarr; A.divv = ctx->d_divv; A.wlinv = ctx->d_wlinv;
  A.tempinv = in->tempinv; A.sig = in->sig; A.capgrey = in->capgrey; A.opaclump = in->opaclump;
  A.emitprob = in->emitprob; A.cap = in->cap; A.tauddmc = in->tauddmc; A.taulump = in->taulump;
  A.T = T;
  A.cellmap = ctx->nmodel > 1 ? ctx->d_cellmap : nullptr;
  A.fp64 = fp64;
  launch_tables(ctx->stream, nx, A);
  return cuda_check(ctx, cudaGetLastError(), "cell tables launch");
}

}  // namespace slg

namespace slg {
// Launch of cell_tables_kernel on caller-provided tables and stream (used by
// the entry point that allocates nothing).
int launch_cell_tables_raw(cudaStream_t st, int nx, int ng, int nep, int nepg, const double* xarr,
                           const double* vxarr, const double* divv, const double* wlinv,
                           const slg_transport_in* in, const CellTables& T) {
  TabArgs A;
  A.nx = nx; A.ng = ng; A.nep = nep; A.nepg = nepg;
  A.xarr = xarr; A.vxarr = vxarr; A.divv = divv; A.wlinv = wlinv;
  A.tempinv = in->tempinv; A.sig = in->sig; A.capgrey = in->capgrey; A.opaclump = in->opaclump;
  A.emitprob = in->emitprob; A.cap = in->cap; A.tauddmc = in->tauddmc; A.taulump = in->taulump;
  A.T = T;
  launch_tables(st, nx, A);
  return cudaGetLastError() == cudaSuccess ? SLG_OK : SLG_ERR_CUDA;
}
}  // namespace slg
