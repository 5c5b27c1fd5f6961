// slg_device.cuh -- device-side constants and helpers shared by the kernels.
//
// Physical constants are those of physconstmod.f:11-51; derived constants are
// written with the Fortran expression order so that the FP64 kernels round
// like the reference (integer powers as explicit products, no FMA contraction:
// the FP64 translation units are compiled with -fmad=false).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace slg {

constexpr double pc_acoef = 7.5657e-15;
constexpr double pc_pi = 3.1415926535897932385;
constexpr double pc_pi2 = 2.0 * pc_pi;
constexpr double pc_pi4 = 4.0 * pc_pi;
constexpr double pc_c = 2.997924562e10;
constexpr double pc_kb = 1.3806505e-16;
constexpr double pc_me = 9.1093826e-28;
constexpr double pc_h = 6.6260693e-27;
constexpr double pc_e = 4.80325e-10;
constexpr double pc_rydberg = 1.0973731534e5;
constexpr double pc_dext = 0.7104;
constexpr double pc_ev = 1.60217653e-12;
constexpr double pc_ang = 1e-8;
constexpr double pc_mbarn = 1e-18;
constexpr double pc_amu = 1.66053886e-24;

constexpr double cinv = 1.0 / pc_c;
constexpr double pi_4th = (pc_pi * pc_pi) * (pc_pi * pc_pi);
constexpr double hck = pc_h * pc_c / pc_kb;              // groupmod.f:110
constexpr double ftpi4 = 15.0 / pi_4th;                   // groupmod.f:109
constexpr double ftpi4r = 15.0 / (4.0 * pi_4th);          // groupmod.f:290
constexpr double planck_c1 = 2.0 * pc_h * (pc_c * pc_c);  // physconstmod.f:87
constexpr double planck_c2 = pc_h * pc_c / pc_kb;         // physconstmod.f:88
constexpr double pc_hc = pc_h * pc_c;
constexpr double e2c = pc_e * pc_e;
constexpr double e4c = e2c * e2c;
constexpr double e6c = e4c * e2c;
constexpr double c2c = pc_c * pc_c;
constexpr double c4c = c2c * c2c;
constexpr double cthomson = 8.0 * pc_pi * e4c / (3.0 * (pc_me * pc_me) * c4c);  // physical_opacity.f:51

// ---- exp by Tang's table-driven method (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15 (1989) 144-157), for the opacity build's inner
// loops, whose one exp per line-shell term is their binding work:
//   x = (64 m + j + f) ln2/64,  |f| <= 1/2,  exp(x) = 2^m 2^(j/64) 2^(f/64),
// 2^(j/64) from a 64-entry table and 2^(f/64) - 1 by its Taylor polynomial of
// degree 5 (truncation below 4e-17 relative), in the form exp(-chi h) with one h
// for many chi, chi in single precision.  The constants and the table are the
// output of csrc/exp_table.py.  (A 256-entry table with a degree-4 polynomial
// saves one FMA per exp but was slower in the opacity kernels.)
constexpr int kExpTabN = 64;
constexpr double kExpInvL = 92.33248261689366;           // 64 / ln 2
constexpr double kExpInvLLo = 1.3027375194195861e-15;    // 64 / ln 2 - kExpInvL
// 2^(j/64), j = 0..63, correctly rounded
static __constant__ double kExp2Tab[kExpTabN] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951,
};

// The division of chi h by ln2/64 is made once per h, in two parts (ExpArg), so
// that n = 64 m + j (the nearest integer of -chi h 64/ln2, by adding and taking
// off 1.5 2^52: the low 32 bits of that sum are n) and f come from one fused
// multiply-add each and f's second part from another.  The
// table is spread over kExpCopies interleaved copies, one per bank pair of a
// half warp, so that no lookup conflicts (random lookups of one copy took about
// six wavefronts), with j << 14 taken off entry j's high word: adding n << 14 to
// it then scales by 2^m and takes the entry's j off again, in one integer
// operation.  The constants come as a kernel argument (ExpConst), which FP64
// instructions read as an operand; as literals they cost moves in the loop.
// Eleven FP64 operations with the caller's multiply-add.  Valid for chi h in
// [-700, 700] (not checked).
struct ExpArg {
  double hi, lo;  // -h 64/ln2
};
constexpr int kExpCopies = 16;                         // one per bank pair of a half warp
struct ExpConst {
  double round = 6755399441055744.0;  // 1.5 * 2^52
  // (ln2/64)^k / k!
  double c1 = 0.010830424696249145, c2 = 5.86490495505617e-05, c3 = 2.1173137155464776e-07,
         c4 = 5.732851688640402e-10, c5 = 1.2417843701716925e-12;
};
__device__ __forceinline__ ExpArg exp_arg(double h) {
  const double hi = -h * kExpInvL;
  return ExpArg{hi, fma(-h, kExpInvLLo, fma(-h, kExpInvL, -hi))};
}
// mine: the byte offset (exp_table_mine) of the caller's copy in s_tab.
__device__ __forceinline__ double exp_scaled(double chi, const ExpArg& a, const ExpConst& C, const double* s_tab,
                                             uint32_t mine) {
  const double big = fma(chi, a.hi, C.round);
  const uint32_t ni = (uint32_t)__double2loint(big);
  const double n = big - C.round;
  const double f = fma(chi, a.lo, fma(chi, a.hi, -n));
  double p = fma(f, C.c5, C.c4);
  p = fma(f, p, C.c3);
  p = fma(f, p, C.c2);
  p = fma(f, p, C.c1);
  p = p * f;
  constexpr uint32_t kMask = 8u * kExpCopies * (kExpTabN - 1);
  const double t = *reinterpret_cast<const double*>(reinterpret_cast<const char*>(s_tab) +
                                                    (((ni * (8u * kExpCopies)) & kMask) | mine));
  const double s = __hiloint2double((int)((uint32_t)__double2hiint(t) + (ni << 14)), __double2loint(t));
  return fma(s, p, s);
}
__device__ __forceinline__ uint32_t exp_table_mine() { return (threadIdx.x & (kExpCopies - 1)) * 8u; }
// Fills a block's spread table (kExpTabN * kExpCopies doubles; call from every
// thread, then __syncthreads()).
__device__ inline void exp_table_spread(double* s_tab) {
  for (int k = threadIdx.x; k < kExpTabN * kExpCopies; k += blockDim.x) {
    const int j = k / kExpCopies;
    const double t = kExp2Tab[j];
    s_tab[k] = __hiloint2double(__double2hiint(t) - (j << 14), __double2loint(t));
  }
}
constexpr double ff_c1a = 4.0 * e6c / (3.0 * pc_h * pc_me * c4c);              // physical_opacity.f:32
constexpr double ff_c1b = pc_pi2 / (3.0 * pc_me * pc_h * pc_c);                 // argument of its sqrt
// Fortran `1.0/3.0` is a real*4 quotient promoted to real*8 as an exponent.
constexpr double third_r4 = (double)(1.0f / 3.0f);

constexpr int FF_NU = 81, FF_NGG = 41;

__host__ __device__ inline double sq(double x) { return x * x; }
__host__ __device__ inline double cube(double x) { return x * x * x; }
__host__ __device__ inline double pow4(double x) { double t = x * x; return t * t; }
__host__ __device__ inline double pow5(double x) { double t = x * x; return t * t * x; }

// MISC/binsrch.f90:3-77.  arr holds n values; returns the 1-based interval
// index (clamped to 1..n-1 unless widerange), -1 for invalid input.
__device__ inline int binsrch(double x, const double* __restrict__ arr, int n, bool widerange) {
  if (n == 2) {
    int r;
    if (x >= arr[0] && x <= arr[1]) r = 1;
    else if (x < arr[0]) r = 0;
    else if (x > arr[1]) r = n;
    else return -1;
    if (!widerange) r = 1;
    return r;
  }
  int imin = 1, imax = n, imid = (n + 1) / 2;
  while (imax - imin > 1) {
    const double amin = arr[imin - 1], amid = arr[imid - 1], amax = arr[imax - 1];
    if (x >= amin && x < amid) {
      imax = imid;
      imid = (imax + imin) / 2;
    } else if (x >= amid && x <= amax) {
      imin = imid;
      imid = (imax + imin) / 2;
    } else {
      if (x < arr[0]) { imin = 0; imid = 0; break; }
      else if (x > arr[n - 1]) { imin = n; imid = n; break; }
      else return -1;
    }
  }
  if (imid != imin) imid = -1;
  if (!widerange) {
    imid = imid > n - 1 ? n - 1 : imid;
    imid = imid < 1 ? 1 : imid;
  }
  return imid;
}

// groupmod.f:99-120 (specint0); ig is 1-based, wlinv holds grp_wlinv(1:ng+1)
__device__ inline double specint0(double tempinv, const double* __restrict__ wlinv, int ig) {
  double x = hck * tempinv;
  const double dx = x * fabs(wlinv[ig] - wlinv[ig - 1]);
  x = x * 0.5 * (wlinv[ig] + wlinv[ig - 1]);
  if (x >= 300.0) x = 300.0;
  return ftpi4 * dx * cube(x) / (exp(x) - 1.0);
}

// groupmod.f:123-143
__device__ inline double dopspeccalc(double tempinv, const double* __restrict__ wlinv, int ig) {
  double x = hck * tempinv;
  x = x * wlinv[ig];
  if (x >= 300.0) x = 300.0;
  return ftpi4 * pow4(x) / (exp(x) - 1.0);
}

// Integrand of specintv, groupmod.f:263-270
__device__ inline double fplanck(double x) {
  if (x >= 300.0) return 27000000.0 / (exp(300.0) - 1.0);
  return cube(x) / (exp(x) - 1.0);
}
// Integrand of spectintv, groupmod.f:395-402
__device__ inline double fross(double x) {
  if (x >= 300.0) {
    const double e3 = exp(300.0);
    return (8100000000.0 * e3) / sq(e3 - 1.0);
  }
  const double ex = exp(x);
  return (pow4(x) * ex) / sq(ex - 1.0);
}
// One element k (0-based, group offset+k) of specintv mode 0 (groupmod.f:189-198):
// x = hck*tempinv*wlinv, ss = ftpi4*|x2-x1|*f((x1+x2)/2).
__device__ inline double specintv_elem(double hct, const double* __restrict__ wlinv, int g0) {
  const double x1 = hct * wlinv[g0], x2 = hct * wlinv[g0 + 1];
  return ftpi4 * fabs(x2 - x1) * fplanck(0.5 * (x2 + x1));
}
__device__ inline double spectintv_elem(double hct, const double* __restrict__ wlinv, int g0) {
  const double x1 = hct * wlinv[g0], x2 = hct * wlinv[g0 + 1];
  double s = ftpi4r * fabs(x2 - x1) * fross(0.5 * (x2 + x1));
  return s != s ? 0.0 : s;  // groupmod.f:390-392
}

// specintv_elem and spectintv_elem of one group (the same values) from one exp.
__device__ inline void spec_weights(double hct, const double* __restrict__ wlinv, int g0, double& w, double& wr) {
  const double x1 = hct * wlinv[g0], x2 = hct * wlinv[g0 + 1];
  const double xm = 0.5 * (x2 + x1), ax = fabs(x2 - x1);
  double fp, fr;
  if (xm >= 300.0) {
    fp = fplanck(xm);
    fr = fross(xm);
  } else {
    const double ex = exp(xm), d = ex - 1.0;
    fp = cube(xm) / d;
    fr = (pow4(xm) * ex) / sq(d);
  }
  w = ftpi4 * ax * fp;
  const double s = ftpi4r * ax * fr;
  wr = s != s ? 0.0 : s;  // groupmod.f:390-392
}

// Sums over the TPC threads (32: a warp; else the whole block) that share a
// cell; every thread gets them.  sh: N * TPC / 32 doubles of the block (TPC > 32).
template <int TPC, int N>
__device__ inline void cell_sum(double* v, double* sh) {
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = v[k] + __shfl_xor_sync(0xffffffffu, v[k], o);
  if (TPC == 32) return;
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) sh[k * (TPC / 32) + (threadIdx.x >> 5)] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    v[k] = sh[k * (TPC / 32)];
#pragma unroll
    for (int w = 1; w < TPC / 32; ++w) v[k] = v[k] + sh[k * (TPC / 32) + w];
  }
}

// The values of cell_sum<32, N> where a block formed a cell's terms: term k of
// group g at part[k * ld + g], N at most eight.  Warp k adds term k in a warp's
// order; every thread of the block gets the sums.  sh: N doubles of the block.
template <int N>
__device__ inline void cell_sum_of_block(const double* part, int ld, int ng, double* v, double* sh) {
  __syncthreads();
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k < N) {
    double a[1] = {0.0};
    for (int g = lane; g < ng; g += 32) a[0] = a[0] + part[k * ld + g];
    cell_sum<32, 1>(a, nullptr);
    if (lane == 0) sh[k] = a[0];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = sh[j];
}

// physconstmod.f:79-93
__device__ inline double planck(double wl, double temp) {
  double b = 1.0 / (wl * temp);
  if (planck_c2 * b >= 300.0) b = 300.0 / planck_c2;
  return planck_c1 * pow5(temp * b) / (exp(planck_c2 * b) - 1.0);
}

// Philox4x32-10 (Salmon, Moraes, Dror & Shaw, SC'11).
struct u32x4 { uint32_t a, b, c, d; };
__device__ inline u32x4 philox4x32_10(u32x4 ctr, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    // one 32 x 32 -> 64-bit multiply gives both halves
    const uint64_t p0 = (uint64_t)0xD2511F53u * ctr.a, p1 = (uint64_t)0xCD9E8D57u * ctr.c;
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    ctr = u32x4{hi1 ^ ctr.b ^ k0, lo1, hi0 ^ ctr.d ^ k1, lo0};
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return ctr;
}
// The same rounds kept out of line for the event loops, which draw from
// many places: one copy of the rounds instead of one per call site keeps the
// loop within the instruction cache.  Same results as philox4x32_10.
static __device__ __noinline__ u32x4 philox4x32_10_call(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                        uint32_t k0, uint32_t k1) {
  return philox4x32_10(u32x4{c0, c1, c2, c3}, k0, k1);
}
__device__ inline double u52_to_unit(uint32_t w0, uint32_t w1) {
  const uint64_t m = ((uint64_t)w0 << 20) | (w1 >> 12);
  return ((double)m + 0.5) * 0x1p-52;
}

// (m + 1/2) 2^-52 of the 52-bit integer m made of two words: 1 + m 2^-52 (m as
// the mantissa under the exponent of 1) minus 1 - 2^-53, exact (the result has
// at most 53 bits and both operands lie in [1/2, 2)).  The same value as
// u52_to_unit without an integer conversion.
__device__ inline double u52_from_bits(uint32_t w0, uint32_t w1) {
  return __hiloint2double((int)(0x3ff00000u | (w0 >> 12)), (int)((w0 << 20) | (w1 >> 12))) - (1.0 - 0x1p-53);
}

// Per-particle stream: draw k uses counter (k/2, pid, stream), words (0,1) for
// even k and (2,3) for odd k; the odd half is kept for the next draw.
struct PhiloxStream {
  uint32_t k0, k1, pid_lo, pid_hi, stream;
  uint32_t k;
  uint32_t w2, w3;
  __device__ inline void init(uint64_t seed, uint64_t pid, uint32_t s) {
    k0 = (uint32_t)seed; k1 = (uint32_t)(seed >> 32);
    pid_lo = (uint32_t)pid; pid_hi = (uint32_t)(pid >> 32);
    stream = s; k = 0;
  }
  __device__ inline double draw() {
    double r;
    if ((k & 1u) == 0u) {
      const u32x4 o = philox4x32_10_call(k >> 1, pid_lo, pid_hi, stream, k0, k1);
      w2 = o.c; w3 = o.d;
      r = u52_to_unit(o.a, o.b);
    } else {
      r = u52_to_unit(w2, w3);
    }
    ++k;
    return r;
  }
};

// The same stream for the FP64 event loop, as a queue of up to three draws.
// begin_event(), called where the warp's lanes are converged, makes one block
// for every lane that holds fewer than two; a third draw of an event makes one
// more block in place for the lanes that ran out.  (With a block made wherever
// a lane's half block ran out, lanes out of step ran the ten rounds at every
// draw site.)  k0, k1 are the key; pid the particle; nb the next block.
struct PhiloxEventStream {
  uint32_t nb, avail;
  uint32_t q[6];
  __device__ inline void init() { nb = 0; avail = 0; }
  __device__ inline void begin_event(uint32_t k0, uint32_t k1, uint64_t pid, uint32_t stream) {
    if (avail >= 2u) return;
    const u32x4 o = philox4x32_10(u32x4{nb, (uint32_t)pid, (uint32_t)(pid >> 32), stream}, k0, k1);
    ++nb;
    if (avail == 0u) {
      q[0] = o.a; q[1] = o.b; q[2] = o.c; q[3] = o.d;
    } else {
      q[2] = o.a; q[3] = o.b; q[4] = o.c; q[5] = o.d;
    }
    avail += 2u;
  }
  __device__ inline double draw(uint32_t k0, uint32_t k1, uint64_t pid, uint32_t stream) {
    if (avail == 0u) {
      const u32x4 o = philox4x32_10_call(nb, (uint32_t)pid, (uint32_t)(pid >> 32), stream, k0, k1);
      ++nb;
      q[0] = o.a; q[1] = o.b; q[2] = o.c; q[3] = o.d;
      avail = 2u;
    }
    const double r = u52_from_bits(q[0], q[1]);
    q[0] = q[2]; q[1] = q[3]; q[2] = q[4]; q[3] = q[5];
    --avail;
    return r;
  }
};
// One particle's draws: the queue with the particle's key and number bound.
struct EventDraws {
  PhiloxEventStream& s;
  uint32_t k0, k1, stream;
  uint64_t pid;
  __device__ inline double draw() { return s.draw(k0, k1, pid, stream); }
};

__device__ inline uint64_t fnv_mix(uint64_t h, int32_t v) {
  const uint32_t u = (uint32_t)v;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    h ^= (u >> (8 * b)) & 0xffu;
    h *= 1099511628211ull;
  }
  return h;
}

}  // namespace slg
