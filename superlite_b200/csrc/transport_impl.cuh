// transport_impl.cuh -- device bodies of one IMC event (transport11) and one
// DDMC event (diffusion11) on a particle held in registers.
//
// Reference: TRANSPORT1/transport11.f90:3-515, TRANSPORT1/diffusion11.f90:3-633,
// GRID/emitgroup.f:3-54.  Arithmetic follows the Fortran expression order;
// the resolved-group scans of diffusion11 and the walk of emitgroup are
// searches over the per-cell running sums built by cell_tables_kernel
// (grid.cu), which hold the very partial sums the scans would form, and the
// DDMC branch probabilities of a (shell, group) are read from the table of
// ddmc_rate_kernel (grid.cu), which evaluates the reference's expressions once
// per entry instead of once per event.
#pragma once
#include "slg_device.cuh"
#include "slg_internal.h"

namespace slg {

struct TrnArgs {
  int nx, ng, nep, nepg;
  const double *xarr, *vxarr, *divv, *wl, *wlinv, *tempinv, *sig, *capgrey, *emitprob, *opaclump;
  const float* cap;
  double tauddmc, taulump;
  int puretran, noampfact, errorfatal, thm_aniso, dogrdtally;
  long long max_steps;
  CellTables T;
  slg_packet* prt;
  int32_t* isvacant;
  long long npart;
  uint64_t seed;
  double *tally, *jrad, *eamp;
  int32_t* methodswap;
  TransportAcc* acc;
  uint64_t* trace_hash;
  int32_t* trace_nstep;
  const unsigned long long* epoch = nullptr;  // replay counter of a captured graph
  int nmodel = 1;                             // models (read by the mixed-precision kernel)
  int smem_cells = 0;                         // tally cells kept in shared memory (mixed kernel; 0: global)
  const ModelDesc* models = nullptr;
  const MixCell* mcell = nullptr;  // per-cell records (mixed-precision kernel)
  // mixed-precision kernel: per (cell, group) DDMC branch rates of an unlumped
  // group, {doplump, opacleak(1), opacleak(2), (1 - emitlump) caplump}, with
  // sentinels and neighbour flags (see mix_rate_kernel); per cell the emission
  // CDF over groups divided by capgrey, and its guide table (T.fine_m ranges per
  // cell)
  const float4* mrate = nullptr;
  const float* emit32 = nullptr;
  const short2* eguide = nullptr;
};

struct Ptcl {
  double x, mu, e, e0, wl, vx;
  int ix, ig, itype, stat, idist;  // ic == ix (1-D, no void cells)
  int lumped;  // DDMC: known to be in a lumped group of its shell
};

// The particle's model: shells nx, first cell co (0-based over every model's
// cells), first shell edge xo of xarr/vxarr.  A one-model grid is {A.nx, 0, 0}.
// ix/ic inside the event bodies stay 1-based shells of the particle's model;
// per-cell arrays are read at co + ic, edges at xo + ix.
struct MView {
  int nx, co, xo;
};

// The ndist histogram of one particle's last events: seven eight-bit counts in
// one register pair (idist -4 and -3 share the first bin as in the reference's
// ndist(-3:7); -1, 5, 6 and 7 do not occur), added to the block's counters
// every 128 events and at the particle's end.  A shared-memory add per event
// and distinct bin put an atomic's latency into every event.
__device__ inline int ndist_slot(int idist) { return idist < -2 ? 0 : (idist == -2 ? 1 : idist + 2); }
__device__ inline void ndist_flush(unsigned long long* s_ndist, unsigned long long& nd8) {
#pragma unroll
  for (int b = 0; b < 7; ++b) {
    const unsigned n = (unsigned)(nd8 >> (8 * b)) & 0xffu;
    if (n) atomicAdd(&s_ndist[b < 2 ? b : b + 1], (unsigned long long)n);
  }
  nd8 = 0;
}

// First entry of running-sum table `table` (0 dop, 1 left, 2 right, 3 scat; a:
// the cell's n entries) of cell `cell` (0-based over all models) whose sum
// exceeds r, else the last one -- the position a linear scan of the reference
// stops at; the sums are non-decreasing.  Searched in the range of the cell's
// guide table.  Returns the entry's info.
__device__ inline int cdf_search(const CellTables& T, int table, int cell, const CdfEntry* __restrict__ a, int n,
                                 double r) {
  int lo = 0, hi = n;
  if (T.fine) {
    const short2 g = __ldg(T.fine + ((size_t)cell * kFineTables + table) * T.fine_m + (int)(r * (double)T.fine_m));
    lo = g.x;
    hi = g.y;
  }
  while (hi - lo > 2) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(&a[mid].sum) <= r) lo = mid + 1;
    else hi = mid;
  }
  // the answer is lo, lo + 1 or lo + 2 = hi
  const int top = min(hi, n - 1);
  const double2* p = reinterpret_cast<const double2*>(a);
  const double2 e0 = __ldg(p + min(lo, top)), e1 = __ldg(p + min(lo + 1, top)), e2 = __ldg(p + top);
  double y = e0.y;
  if (lo < hi && e0.x <= r) y = e1.y;
  if (lo + 1 < hi && e1.x <= r) y = e2.y;
  return __double2loint(y);
}

// First position q in [lo, hi] with a[q] > r (hi if none), at most n - 1, for
// a non-decreasing a; 8-ary: the 7 probes of a round are independent loads.
// The mixed-precision loop's searches: its guide narrows the search over the
// FP32 running sums.  Where rounding
// to FP32 moves a sum across r the answer may differ from the FP64 search by
// one position (the result stays within the guide's range).
__device__ inline int first_gt_range32(const float* __restrict__ a, int lo, int hi, int n, float r) {
  while (hi - lo > 8) {
    const int step = (hi - lo) >> 3;
    float v[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) v[j] = __ldg(a + lo + (j + 1) * step);
    int c = 0;
#pragma unroll
    for (int j = 0; j < 7; ++j) c += v[j] <= r;
    const int nlo = c == 0 ? lo : lo + c * step + 1;
    const int nhi = c == 7 ? hi : lo + (c + 1) * step;
    lo = nlo;
    hi = nhi;
  }
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = lo + j < hi ? __ldg(a + lo + j) : 0.0f;
  int c = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) c += (lo + j < hi) && v[j] <= r;
  const int q = lo + c;
  return q < n ? q : n - 1;
}
__device__ inline int cdf_search32(const CellTables& T, int table, int cell, const float* __restrict__ a, int n,
                                   float r) {
  if (!T.guide) return first_gt_range32(a, 0, n, n, r);
  const int16_t* g = T.guide + ((size_t)cell * 4 + table) * (T.guide_m + 1);
  const int k = (int)(r * (float)T.guide_m);  // exact: guide_m is a power of two and r < 1
  return first_gt_range32(a, g[k], g[k + 1], n, r);
}

__device__ inline double CAPd(const TrnArgs& A, int ig, int ic) {
  return (double)__ldg(A.cap + (size_t)(ic - 1) * A.ng + (ig - 1));
}
__device__ inline double dxv(const double* X, int i) { return X[i] - X[i - 1]; }

// GRID/emitgroup.f:3-54 (LTE) for the 0-based cell gc: the group of draw r from
// the shell's emission thresholds (CellTables::emitcum, see cell_tables_kernel)
// -- the number of thresholds not above r * capgrey, plus one -- searched in
// the range that the guide table gives for r (the whole table without one).
__device__ inline int emitgroup_dev(const TrnArgs& A, double r, int gc, double capgrey) {
  const double r1 = r * capgrey;
  const double* t = A.T.emitcum + (size_t)gc * A.ng;
  int lo, hi;
  if (A.T.fine) {
    const short2 g =
        __ldg(A.T.fine + ((size_t)gc * kFineTables + 4) * A.T.fine_m + (int)(r * (double)A.T.fine_m));
    lo = g.x;
    hi = g.y;
  } else {
    const int one = emit_only_group(A.nep, A.nepg, A.ng, r1 != r1);
    if (one) return one;
    lo = 0;
    hi = emit_last_group(A.nep, A.nepg, A.ng) - 1;
  }
  while (hi - lo > 2) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(t + mid) > r1) hi = mid;
    else lo = mid + 1;
  }
  const double v0 = lo < hi ? __ldg(t + lo) : 0.0, v1 = lo + 1 < hi ? __ldg(t + lo + 1) : 0.0;
  return 1 + lo + (int)(lo < hi && !(v0 > r1)) + (int)(lo + 1 < hi && !(v1 > r1));
}

// a / 3 correctly rounded, by Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990): with y = RN(1/3), q = RN(a y) is within an ulp of a/3, its
// remainder is exact, and RN(q + rem y) is the rounded quotient (results in
// the normal range; an infinite or NaN a, whose remainder is NaN, is returned).
__device__ __forceinline__ double third_of(double a) {
  constexpr double y = 1.0 / 3.0;
  const double q = a * y;
  const double r = fma(fma(-3.0, q, a), y, q);
  return r == r ? r : a;
}

// fabs(a) / pc_c >= 0.1 (transport11.f90:159) as a comparison with the smallest
// double whose rounded quotient by pc_c reaches 0.1 (the quotient is monotone
// in a, so the two tests agree for every a, NaN included).
constexpr double newton_velocity_threshold() {
  double t = 0.1 * pc_c;
  const double ulp = 4.76837158203125e-07;  // of numbers in [2^31, 2^32), which t is
  while (t / pc_c >= 0.1) t -= ulp;
  while (!(t / pc_c >= 0.1)) t += ulp;
  return t;
}
constexpr double kNewtonVelocity = newton_velocity_threshold();
static_assert(kNewtonVelocity > 2147483648.0 && kNewtonVelocity < 4294967296.0, "spacing of the search");

// One IMC event, transport11.f90:3-515.  The two sides of a shell share one
// code path, so lanes that cross either way stay together.
template <class RNG>
__device__ inline void transport11_dev(const TrnArgs& A, const MView& v, Ptcl& p, RNG& rng, double& eraddens,
                                       double& eamp, double& jrad, double& totevelo, int& ierr) {
  int& ix = p.ix;
  int& ig = p.ig;
  double& x = p.x;
  double& mu = p.mu;
  double& e = p.e;
  double& e0 = p.e0;
  double& wl = p.wl;
  double& vx = p.vx;
  const int gc = v.co + ix - 1;          // 0-based cell over all models
  const TrnCell& R = A.T.cell[gc];
  ierr = 0;
  eraddens = 0.0;
  eamp = 0.0;
  jrad = 0.0;
  const double capc = CAPd(A, ig, gc + 1);
  double elabfact = 1.0 - mu * vx * cinv;
  const double elabfactold = elabfact;
  const double far = R.far;
  const double Xa = R.xa, Xb = R.xb;
  // outward unless the chord meets the inner shell (:95-103); for mu >= 0 and
  // x >= Xa the root is of a number >= 0, so mu is not below its negative.  The
  // two sides share one root: sqrt(..) - mu x outward, sqrt(..) + mu x inward.
  const bool outer = ix == 1 || (mu >= 0.0 && x >= Xa) || mu >= -sqrt(1.0 - sq(Xa / x));
  const int ixnext = outer ? ix + 1 : ix - 1;
  const double db = fabs(sqrt(sq(outer ? Xb : Xa) - (1.0 - sq(mu)) * sq(x)) + (outer ? -mu : mu) * x);
  if (db != db) { ierr = 1; return; }
  const double sigc = R.sig;
  double dthm, dcol, ddop, r1, r2, help;
  if (sigc > 0.0) {
    r1 = rng.draw();
    dthm = -log(r1) / (elabfact * sigc);
  } else {
    dthm = far;
  }
  if (capc <= 0.0) {
    dcol = far;
  } else {
    r1 = rng.draw();
    dcol = -log(r1) / (elabfact * capc);
  }
  const double dvdr = R.dvdr;
  const double vhelp = R.vhelp;
  if (fabs(vx - vhelp) >= kNewtonVelocity) {
    // Newton-Raphson Doppler distance (transport11.f90:159-199)
    const double epstol = 1e-3;
    int it = 0;
    double shelp = db;
    double xhelp = sqrt(sq(x) + sq(shelp) + 2.0 * shelp * x * mu);
    double muhelp = (mu * x + shelp) / xhelp;
    double phi = dvdr * mu * x - pc_c * (1.0 - wl * A.wlinv[ig]) + vhelp * muhelp + dvdr * shelp;
    double dphi = dvdr + vhelp * (1.0 - sq(muhelp)) / xhelp;
    ddop = shelp - phi / dphi;
    while ((fabs(ddop - shelp) > ddop * epstol) && it < 100) {
      it = it + 1;
      shelp = ddop;
      xhelp = sqrt(sq(x) + sq(shelp) + 2.0 * shelp * x * mu);
      muhelp = (mu * x + shelp) / xhelp;
      if (dvdr > 0.0 && ig < A.ng) {
        phi = dvdr * mu * x - pc_c * (1.0 - wl * A.wlinv[ig]) + vhelp * muhelp + dvdr * shelp;
      } else if (dvdr < 0.0 && ig > 1) {
        phi = dvdr * mu * x - pc_c * (1.0 - wl * A.wlinv[ig - 1]) + vhelp * muhelp + dvdr * shelp;
      } else {
        ddop = far;
        break;
      }
      dphi = dvdr + vhelp * (1.0 - sq(muhelp)) / xhelp;
      ddop = shelp - phi / dphi;
    }
    if (ddop <= 0.0 || it == 100) ddop = far;
  } else {
    if (dvdr > 0.0 && ig < A.ng) {
      ddop = R.dopc * (elabfact - wl * A.wlinv[ig]);
    } else if (dvdr < 0.0 && ig > 1) {
      ddop = R.dopc * (elabfact - wl * A.wlinv[ig - 1]);
    } else {
      ddop = far;
    }
    if (ddop < 0.0) ddop = far;
  }
  // minloc over [dcol,dthm,ddop,db]; ties resolve to the first
  double d = dcol;
  int im = 1;
  if (dthm < d) { d = dthm; im = 2; }
  if (ddop < d) { d = ddop; im = 3; }
  if (db < d) { d = db; im = 4; }
  p.idist = im;
  if (dcol != dcol || dthm != dthm || ddop != ddop) { ierr = 3; return; }
  if (d < 0.0) { ierr = 4; return; }
  const double xold = x;
  x = sqrt(sq(x) + sq(d) + 2.0 * d * x * mu);
  vx = (R.vxa * (Xb - x) + R.vxb * (x - Xa)) / R.dist;
  if (x == 0.0) mu = 1.0;
  else mu = (xold * mu + d) / x;
  eraddens = e * sq(elabfact) * d * cinv;
  jrad = pc_c * eraddens;
  elabfact = 1.0 - mu * vx * cinv;
  if (x < R.x0) {
    x = R.x0;
    vx = A.vxarr[v.xo];
    ix = 1;
    r1 = rng.draw();
    mu = 1.0 - r1;
    return;
  }
  if (d == dthm || d == dcol) {
    r1 = rng.draw();
    if (d == dthm && A.thm_aniso) {
      // transport11.f90:259-281 (experimental)
      const double s = sqrt(1.0 + 16.0 * pow(r1 - 0.5, 2.0));
      const double mutemp = pow(4.0 * r1 - 2.0 + s, 1.0 / 3.0) - pow(s - (4.0 - 2.0 * r1), 1.0 / 3.0);
      const double mh = mutemp;
      const double B = 2.0 * mutemp * mh;
      const double Cc = sq(mutemp) + sq(mh) - 1.0;
      const double munew1 = (-B + sqrt(sq(B) - 4.0 * Cc)) / 2.0;
      const double munew2 = (-B - sqrt(sq(B) - 4.0 * Cc)) / 2.0;
      const bool ok1 = munew1 <= 1.0 && munew1 >= -1.0, ok2 = munew2 <= 1.0 && munew2 >= -1.0;
      if (ok1 && ok2) mu = r1 < 0.5 ? munew1 : munew2;
      else if (ok1) mu = munew1;
      else if (ok2) mu = munew2;
      else mu = 1.0 - 2.0 * r1;
    } else {
      mu = 1.0 - 2.0 * r1;
    }
    mu = (mu + vx * cinv) / (1.0 + vx * mu * cinv);
  } else if (d == db) {
    // transport11.f90:290-295.  A grazing exit through the outer edge can leave
    // mu a rounding error below 0; the reference would then index shell nx+1.
    if ((mu >= 0.0 && ix == v.nx) || ixnext > v.nx) { p.stat = 1; return; }
  }
  if (d == dthm) {
    wl = wl * (1.0 - mu * vx * cinv) / elabfact;
    help = elabfact / (1.0 - mu * vx * cinv);
    totevelo = totevelo + e * (1.0 - help);
    e = e * help;
    e0 = e0 * help;
  } else if (d == dcol) {
    r1 = rng.draw();  // drawn and unused in the reference (transport11.f90:313)
    help = elabfact / (1.0 - mu * vx * cinv);
    totevelo = totevelo + e * (1.0 - help);
    e = e * help;
    e0 = e0 * help;
    if (A.ng != 1) {
      r1 = rng.draw();
      ig = emitgroup_dev(A, r1, gc, R.capgrey);
      if (((sigc + CAPd(A, ig, gc + 1)) * R.dist >= A.tauddmc) && !A.puretran) p.itype = 2;
    }
    if (p.itype == 2) {
      totevelo = totevelo + e * vx * mu * cinv;
      e = e * (1.0 - vx * mu * cinv);
      e0 = e0 * (1.0 - vx * mu * cinv);
    } else {
      r1 = rng.draw();
      wl = 1.0 / ((1.0 - r1) * A.wlinv[ig - 1] + r1 * A.wlinv[ig]);
      wl = wl * (1.0 - vx * mu * cinv);
    }
  } else if (d == db) {
    // the outer (:344-394) or inner (:397-458) face
    const bool out = ixnext > ix;
    const double capl = CAPd(A, ig, out ? gc + 2 : gc), sigl = out ? R.sigr : R.sigl;
    const double dxl = out ? R.dxr : R.dxl;
    if ((sigl + capl) * dxl < A.tauddmc || A.puretran) {
      x = out ? Xb : Xa;
      vx = out ? R.vxb : R.vxa;
      ix = ixnext;
    } else {
      mu = (mu - vx * cinv) / (1.0 - vx * mu * cinv);
      if (!out && !A.noampfact && mu < 0.0) {
        help = 1.0 / fabs(mu);
        help = help < 100.0 ? help : 100.0;
        totevelo = totevelo - e * 2.0 * (0.55 * help - 1.25 * fabs(mu)) * vx * cinv;
        const double hm2 = help - 2.0;
        eamp = e * 2.0 * 0.55 * (hm2 > 0.0 ? hm2 : 0.0) * vx * cinv;
        help = help < 2.0 ? help : 2.0;
        e0 = e0 * (1.0 + 2.0 * (0.55 * help - 1.25 * fabs(mu)) * vx * cinv);
        e = e * (1.0 + 2.0 * (0.55 * help - 1.25 * fabs(mu)) * vx * cinv);
      }
      help = (capl + sigl) * dxl;
      help = 4.0 / (3.0 * help + 6.0 * pc_dext);
      r1 = rng.draw();
      if (r1 < help * (1.0 + 1.5 * fabs(mu))) {
        p.itype = 2;
        totevelo = totevelo + e * (1.0 - elabfact);
        e = e * elabfact;
        e0 = e0 * elabfact;
        wl = wl / elabfact;
        ix = ixnext;
      } else {
        r1 = rng.draw();
        r2 = rng.draw();
        const double m = r1 > r2 ? r1 : r2;
        mu = out ? -m : m;
        mu = (mu + vx * cinv) / (1.0 + vx * mu * cinv);
        x = out ? Xb : Xa;
        vx = out ? R.vxb : R.vxa;
      }
    }
  } else if (d == ddop) {
    if (dvdr > 0.0) {
      if (ig < A.ng) {
        ig = ig + 1;
        wl = (A.wl[ig - 1] + 1e-6 * (A.wl[ig] - A.wl[ig - 1])) * elabfactold;
      } else {
        r1 = rng.draw();
        wl = 1.0 / (r1 * A.wlinv[A.ng] + (1.0 - r1) * A.wlinv[A.ng - 1]);
        wl = wl * elabfact;
      }
    } else if (dvdr < 0.0) {
      if (ig > 1) {
        wl = (A.wl[ig - 1] + 1e-6 * (A.wl[ig - 2] - A.wl[ig - 1])) * elabfactold;
        ig = ig - 1;
      } else {
        r1 = rng.draw();
        wl = 1.0 / (r1 * A.wlinv[0] + (1.0 - r1) * A.wlinv[1]);
        wl = wl * elabfact;
      }
    }
    if (((sigc + CAPd(A, ig, gc + 1)) * R.dist >= A.tauddmc) && !A.puretran) {
      p.itype = 2;
      totevelo = totevelo + e * vx * mu * cinv;
      e = e * elabfact;
      e0 = e0 * elabfact;
      wl = wl / elabfact;
    }
  } else {
    ierr = 17;
  }
}

// (shell, group) is IMC: the table's sentinel, the test (sig + cap) dx < tauddmc
__device__ inline bool rate_is_imc(const TrnArgs& A, int gc, int ig) {
  return __double2hiint(__ldg(&A.T.rates[2 * ((size_t)gc * A.ng + (ig - 1))].x)) == kRateImcHi;
}

// One DDMC event, diffusion11.f90:3-633 (LTE).
template <class RNG>
__device__ inline void diffusion11_dev(const TrnArgs& A, const MView& v, Ptcl& p, RNG& rng, double& eraddens,
                                       double& jrad, double& totevelo, int& ierr) {
  const int ng = A.ng;
  int& ix = p.ix;
  int& ig = p.ig;
  double& x = p.x;
  double& mu = p.mu;
  double& e = p.e;
  double& e0 = p.e0;
  double& wl = p.wl;
  double& vx = p.vx;
  const int gc = v.co + ix - 1;          // 0-based cell over all models
  const TrnCell& R = A.T.cell[gc];
  ierr = 0;
  eraddens = 0.0;
  jrad = 0.0;
  const size_t off = (size_t)gc * ng;
  // this group's branch probabilities (:154-278), or the shell's for a lumped group
  double2 ra = make_double2(0.0, 0.0), rb = ra;
  if (!p.lumped) {
    ra = __ldg(A.T.rates + 2 * (off + ig - 1));
    rb = __ldg(A.T.rates + 2 * (off + ig - 1) + 1);
    const int tag = __double2hiint(ra.x);
    if (tag == kRateImcHi) { ierr = 100; return; }
    p.lumped = tag == kRateLumpedHi;
  }
  int glump = 0;
  if (p.lumped) {
    glump = R.nlump;
    ra = make_double2(R.denom, R.pdop);
    rb = make_double2(R.pleft, R.pleak);
  }
  double r1, r2, help;
  r1 = rng.draw();
  const double ddmct = fabs(log(r1) * ra.x * cinv);
  eraddens = e * ddmct;
  jrad = pc_c * eraddens;
  r1 = rng.draw();
  const double divv = R.divv;
  double dv = divv;  // of the shell after the event
  bool to_imc = false;
  p.lumped = 0;
  if (r1 < ra.y) {
    // Doppler shift (:283-355)
    int iiig = ig, info = 0;
    if (glump != 0) {
      r1 = rng.draw();
      info = cdf_search(A.T, 0, gc, A.T.cdf_dop + off, glump, r1);
      iiig = info & 0xffff;
    }
    if (divv >= 0.0) {
      ig = iiig + 1;
      wl = A.wl[ig - 1];
      ig = ig < ng ? ig : ng;
    } else {
      ig = iiig - 1;
      wl = A.wl[ig];
      ig = ig > 1 ? ig : 1;
    }
    p.lumped = info & kInfoLumped;
    to_imc = glump != 0 ? (info & kInfoImc) != 0 : rate_is_imc(A, gc, ig);
  } else if (r1 >= ra.y && r1 < rb.y) {
    // leakage to a neighbour: left (:358-430) or right (:434-545).  Both
    // directions run one code path (same draws, same arithmetic as each
    // branch of the reference) so lanes of a warp leaking either way stay
    // together.
    const bool right = r1 >= rb.x;
    p.idist = right ? -4 : -3;
    if (!right && ix == 1) return;
    if (right && ix == v.nx) {
      // escape through the outer edge (:438-478)
      p.stat = 1;
      r1 = rng.draw();
      r2 = rng.draw();
      mu = r1 > r2 ? r1 : r2;
      if (glump != 0) {
        r1 = rng.draw();
        ig = cdf_search(A.T, 2, gc, A.T.cdf_right + off, glump, r1) & 0xffff;
      }
      r1 = rng.draw();
      wl = 1.0 / (r1 * A.wlinv[ig] + (1.0 - r1) * A.wlinv[ig - 1]);
      x = R.xb;
      vx = R.vxb;
      mu = (mu + vx * cinv) / (1.0 + vx * mu * cinv);
      mu = mu < 1.0 ? mu : 1.0;
      help = 1.0 / (1.0 - mu * vx * cinv);
      totevelo = totevelo + e * (1.0 - help);
      wl = wl / help;
      e = e * help;
      e0 = e0 * help;
      return;
    }
    dv = right ? R.divvr : R.divvl;
    bool imc;
    if (glump != 0) {
      r1 = rng.draw();
      const int info =
          cdf_search(A.T, right ? 2 : 1, gc, (right ? A.T.cdf_right : A.T.cdf_left) + off, glump, r1);
      ig = info & 0xffff;
      p.lumped = info & kInfoLumped;
      imc = (info & kInfoImc) != 0;
    } else {
      imc = rate_is_imc(A, right ? gc + 1 : gc - 1, ig);
    }
    if (imc) {
      p.itype = 1;
      r1 = rng.draw();
      wl = 1.0 / (r1 * A.wlinv[ig] + (1.0 - r1) * A.wlinv[ig - 1]);
      x = right ? R.xb : R.xa;
      vx = right ? R.vxb : R.vxa;
      r1 = rng.draw();
      r2 = rng.draw();
      const double m = r1 > r2 ? r1 : r2;
      mu = right ? m : -m;
      mu = (mu + vx * cinv) / (1.0 + vx * mu * cinv);
      help = 1.0 / (1.0 - vx * mu * cinv);
      totevelo = totevelo + e * (1.0 - help);
      e = e * help;
      e0 = e0 * help;
      wl = wl * (1.0 - vx * mu * cinv);
    }
    ix = right ? ix + 1 : ix - 1;
  } else {
    // effective scattering (:549-620)
    p.idist = -2;
    if (glump == ng) { ierr = 102; return; }
    r1 = rng.draw();
    if (glump == 0) {
      ig = emitgroup_dev(A, r1, gc, R.capgrey);
      to_imc = rate_is_imc(A, gc, ig);
    } else {
      const int info = cdf_search(A.T, 3, gc, A.T.cdf_scat + off, ng - glump, r1);
      ig = info & 0xffff;
      to_imc = (info & kInfoImc) != 0;
    }
    if (to_imc) {
      r1 = rng.draw();
      wl = 1.0 / ((1.0 - r1) * A.wlinv[ig - 1] + r1 * A.wlinv[ig]);
    }
  }
  if (to_imc) {
    // IMC in this shell after a Doppler shift (:336-353) or a scattering
    // (:597-618): the same direction and position draws
    p.itype = 1;
    const double Xa = R.xa, Xb = R.xb;
    r1 = rng.draw();
    mu = 1.0 - 2.0 * r1;
    r1 = rng.draw();
    x = pow(r1 * R.xb3 + (1.0 - r1) * R.xa3, third_r4);
    x = x < Xb ? x : Xb;
    x = x > Xa ? x : Xa;
    vx = (R.vxa * (Xb - x) + R.vxb * (x - Xa)) / R.dist;
    mu = (mu + vx * cinv) / (1.0 + vx * mu * cinv);
    help = 1.0 / (1.0 - vx * mu * cinv);
    totevelo = totevelo + e * (1.0 - help);
    e = e * help;
    e0 = e0 * help;
    wl = wl * (1.0 - vx * mu * cinv);
  }
  if (x < R.x0) { p.stat = 2; return; }
  const double decay = exp(third_of(-dv * ddmct));
  totevelo = totevelo + e * (1.0 - decay);
  e = e * decay;
  e0 = e0 * decay;
}


}  // namespace slg
