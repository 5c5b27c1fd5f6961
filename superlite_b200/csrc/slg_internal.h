// slg_internal.h -- host-side context and launch declarations of libslg.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>
#include "slg.h"

namespace slg {

// A device buffer that grows on demand and is freed with the context.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

// High words of the sentinels in CellTables::rates (quiet NaNs with payloads
// that arithmetic does not produce): the group is IMC in this shell, or one of
// its lumped groups (whose values are the record's).
constexpr int kRateImcHi = 0x7ff8dd01, kRateLumpedHi = 0x7ff8dd02;

// Per-cell record of the FP64 particle loop: what an event reads about its
// shell apart from per-group values, in two 128-byte lines instead of a dozen
// arrays; quotients and powers of the shell alone are formed once here, by the
// event's expressions.
struct alignas(256) TrnCell {
  double xa, xb, vxa, vxb;       // shell edges and edge velocities
  double dist, sig, divv, capgrey;
  double denom, pdop, pleft, pleak;  // the lumped groups' entry of CellTables::rates
  double x0;                     // the model's inner edge
  double far, dvdr, vhelp;       // vhelp = vxa - dvdr xa
  double dopc;                   // 3 c / divv
  double sigl, sigr, dxl, dxr;   // neighbours (0 at the model's ends)
  double divvl, divvr;
  double xa3, xb3;               // cubed edges
  int nlump, pad;
};
static_assert(sizeof(TrnCell) == 256, "TrnCell is two 128-byte lines");

// Entry of a resolved-group running sum: the sum, the group that its position
// resolves to, and in bit 16 whether that group is lumped, in bit 17 whether
// it is IMC, in the shell where the particle continues (for a Doppler shift:
// of the group it shifts to).
struct __align__(16) CdfEntry {
  double sum;
  int info, pad;
};
constexpr int kInfoLumped = 1 << 16, kInfoImc = 1 << 17;

// Device-resident per-cell tables used by the transport kernels (built by
// build_cell_tables from grd_cap, grd_sig, grd_opaclump ...).  All tables
// are cell-major: entry (ic-1)*ng + k.
struct CellTables {
  double* specarr = nullptr;  // specintv mode-0 Planck weights
  int16_t* glumps = nullptr;  // diffusion11.f90:103-124 ordering (1-based groups)
  // resolved-group running sums: for the FP64 loop each entry with the group it
  // resolves to, for the mixed loop (which reads their FP32 copies) the sums alone
  CdfEntry* cdf_dop = nullptr;  // Doppler (:290-314)
  CdfEntry* cdf_left = nullptr; // left leak (:375-398)
  CdfEntry* cdf_right = nullptr;// right leak (:447-460 at ix==nx, :489-511 else)
  CdfEntry* cdf_scat = nullptr; // effective scatter over unlumped groups (:571-584)
  double *sum_dop = nullptr, *sum_left = nullptr, *sum_right = nullptr, *sum_scat = nullptr;
  // emitgroup's thresholds (emitgroup.f:3-54): entry g-1 is the draw (times
  // capgrey) from which group g+1 is emitted, see cell_tables_kernel
  double* emitcum = nullptr;
  // FP64 loop: DDMC branch probabilities per (cell, group), two double2 each
  // {1/R, P(Doppler)}, {P(Doppler) + P(left), P(Doppler) + P(either leak)} with
  // R the sum of the branch rates, or a sentinel in the first word (kRate*Hi);
  // per-cell records
  double2* rates = nullptr;
  TrnCell* cell = nullptr;
  // guide tables of the FP64 loop: fine_m entries per cell and table (four
  // running sums and emitcum), entry k = the range {first, last} of answers for
  // draws in [k, k+1)/fine_m.  fine_m is a power of two (r * fine_m is exact)
  // near ng, so most ranges hold one or two entries and a search is one load
  // of the range and one round of loads (null: search the whole table)
  short2* fine = nullptr;
  int fine_m = 0;
  // per-cell scalars: nlump, emitlump, caplump, doplump, capgreyinv, speclump
  int32_t* nlump = nullptr;
  double* scal = nullptr;     // 8 doubles per cell (see SCAL_*)
  // guide tables of the mixed loop's searches, of the four running sums above
  // (dop, left, right, scat): per cell and table guide_m+1 entries, entry k = number of sums <= k/guide_m,
  // so a draw r in [k, k+1)/guide_m is searched only between entries k and k+1
  // (null: plain search over the whole table).  guide_m is a power of two
  // (so r * guide_m and k / guide_m are exact) near ng/4: a range of a few
  // entries, searched in one round of loads, without a guide larger than the
  // tables it indexes.
  int16_t* guide = nullptr;
  int guide_m = 0;
  // FP32 copies of cdf_dop/left/right/scat for the mixed-precision loop (half
  // the bytes per gather; null when only the FP64 loop runs)
  float *cdf32_dop = nullptr, *cdf32_left = nullptr, *cdf32_right = nullptr, *cdf32_scat = nullptr;
  // the grid that the tables are for, and which loops' tables are in place (each is
  // allocated by the first launch that reads it)
  int nx = 0, ng = 0;
  bool have_fp64 = false, have_mixed = false;
};
// emitgroup's last reachable group, and its constant answer where it has one
// (0: none): one emission bin, or a draw that is not a number (nan).
__host__ __device__ inline int emit_last_group(int nep, int nepg, int ng) {
  const long long n = nep == 1 ? nepg + 1 : (long long)nep * nepg;
  return n < ng ? (int)n : ng;
}
__host__ __device__ inline int emit_only_group(int nep, int nepg, int ng, bool nan) {
  if (nep == 1) return emit_last_group(nep, nepg, ng);
  return nan ? (nepg < ng ? nepg : ng) : 0;
}

constexpr int kFineMax = 2048;
inline int fine_size(int ng) {
  int m = 16;
  while (m < kFineMax && m < ng) m *= 2;
  return m;
}
constexpr int kFineTables = 5;  // dop, left, right, scat, emitcum
constexpr int kGuideMax = 256;
inline int guide_size(int ng) {
  int m = 16;
  while (m < kGuideMax && 4 * m < ng) m *= 2;
  return m;
}

// Per-cell record of the mixed-precision particle loop: everything an event
// reads about its shell except per-group values, in one 128-byte line
// (instead of about ten lines of separate arrays).  Values are the same
// roundings the event code made from the separate arrays.
struct alignas(128) MixCell {
  double xa, xb, vxa, vxb;  // shell edges and edge velocities
  double x0;                // the model's inner edge
  double capgreyinv, tinv;  // 1/capgrey, 1/T
  int nlump, pad;
  float dist, sig, emitlump, caplump, doplump, o1, o2, divv;  // o1, o2: opaclump(1:2) of the lumped groups
  float far, dvdr, sigl, sigr, dxl, dxr, fa, fb;  // neighbours (0 at the model's ends); fa, fb = x^2 / dx3
};
static_assert(sizeof(MixCell) == 128, "MixCell is one 128-byte line");
enum { SCAL_EMITLUMP = 0, SCAL_CAPLUMP, SCAL_DOPLUMP, SCAL_CAPGREYINV, SCAL_SPECLUMP, SCAL_FAR,
       SCAL_DX3, SCAL_DVDR, SCAL_N };

// A result on its way to a host array through the context's pinned block.
struct HostOut {
  void* dst;
  const void* src;
  size_t bytes;
};
constexpr int kHostOut = 16;

// Accumulators written by the transport kernel (device memory).
struct TransportAcc {
  double evelo, eout, sflux;
  unsigned long long npckt, nflux, nimc, nddmc, nswap, nmax, nwarn;
  unsigned long long ndist[11];
  unsigned long long ierr_key;  // (ipart << 32) | ierr, min over particles
  unsigned long long next;      // persistent-kernel work counter
};

// One ejecta model of a multi-model context: particle slots [poff, poff+np),
// cells [co, co+nx) of every per-cell array, shell edges [xo, xo+nx] of
// xarr/vxarr (xo = co + model index).
struct ModelDesc {
  long long poff, np;
  int nx, co, xo, pad;
};

// Random-number key of model m: seed + m * kModelSeedStride (SLG_MODEL_SEED_STRIDE).
constexpr unsigned long long kModelSeedStride = 0x9E3779B97F4A7C15ULL;

}  // namespace slg

struct slg_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  // groups
  int ng = 0, nep = 0, nepg = 0;
  double* d_wl = nullptr;
  double* d_wlinv = nullptr;
  std::vector<double> h_wl;
  // grid
  int nx = 0;
  double* d_xarr = nullptr;
  double* d_vxarr = nullptr;
  double* d_vol = nullptr;
  double* d_divv = nullptr;
  std::vector<double> h_xarr;
  // atomic data
  int nelem = 0, nstage = 0;
  int64_t nline = 0;
  int32_t* d_ion_ni = nullptr;
  std::vector<int32_t> h_ion_ni;
  slg_bbxs* d_bb = nullptr;
  // population rows (slot = (iz-1) nstage + ii-1) that the lines reference:
  // d_lrow_of_slot[slot] = compact row or -1, after them the rows' slots
  int nlrow = 0;
  double line_chimax = 0.0;  // largest chilw of the lines (infinite if any is negative or NaN)
  int16_t* d_lrow_of_slot = nullptr;
  float* d_ph1 = nullptr;
  float* d_ph2 = nullptr;
  double* d_gff = nullptr;
  std::vector<float> h_ph1, h_ph2;
  // ion data of the equation of state: stages, ionisation energies,
  // partition functions and ground-level weights, (nstage, nelem) each
  int eos_nelem = 0, eos_nstage = 0;
  int32_t* d_eos_ni = nullptr;
  double* d_eos_e = nullptr;
  double* d_eos_q = nullptr;
  double* d_eos_g1 = nullptr;
  double* d_amass = nullptr;  // element masses [amu] of the differentiable opacity
  int amass_n = 0;
  // derived per-call scratch
  slg::DevBuf scratch[128];
  slg::CellTables tables;
  // opacity_plan's layouts that are in place (for plan_ngs sub-groups)
  int plan_ngs = 0;
  bool plan_edges = false, plan_bb = false, plan_bf = false;
  slg::TransportAcc* d_acc = nullptr;
  // a host call's small results on their way (capi.cu, down and finish)
  char* h_block = nullptr;                    // pinned, taken by the first such call
  bool host_tried = false;                    // (once)
  size_t host_used = 0;                       // bytes of it that the current call took
  slg::HostOut host_out[slg::kHostOut] = {};  // what finish() copies out of it
  int nhost_out = 0;
  slg::TransportAcc* h_acc = nullptr;  // pinned
  // optional trace (host arrays) for the next particle_advance call
  uint64_t* trace_hash = nullptr;
  int32_t* trace_nstep = nullptr;
  // transport kernel variants until slg_autotune_transport or
  // slg_set_transport_variant choose (-1: by the rules of
  // launch_transport_variant and launch_transport_mixed)
  int trn_variant = -1;
  int mix_variant = -1;
  // transport_out of a queued slg_dev_particle_advance, completed by slg_sync
  slg_transport_out* pending_out = nullptr;
  // models (one for slg_set_grid): host descriptors, device copies, and the
  // per-cell map {local 1-based shell, model nx, model first cell, model}
  int nmodel = 0;
  std::vector<slg::ModelDesc> h_models;
  slg::ModelDesc* d_models = nullptr;
  int4* d_cellmap = nullptr;  // null for a single model
  long long npart_models = 0;  // sum of the models' particle slots (0: one unranged model)
  // running sums of the transport counters over launches (device; they
  // survive graph replays), the replay counter that offsets the random
  // streams of captured launches, and the captured graph
  slg::TransportAcc* d_totals = nullptr;
  unsigned long long* d_epoch = nullptr;
  int capturing = 0;
  int capture_failed = 0;  // a call failed during the open capture
  cudaGraphExec_t graph_exec = nullptr;
  // host copies of the last uploaded source set-up (an unchanged set-up is
  // not uploaded again, so captured steps hold no host copies)
  std::vector<double> src_emit;
  std::vector<int32_t> src_nvol;
  int num_sms = 0;
};

namespace slg {
// Raises kernel `fn`'s dynamic shared-memory limit to `bytes` on the current
// device (the context's: every entry point selects it) the first time a
// launch there needs it; the attribute holds per device, so `mask` keeps one
// bit per device id.
template <class F>
inline void raise_smem_limit(unsigned& mask, int device, F* fn, int bytes) {
  const unsigned bit = device >= 0 && device < 32 ? 1u << device : 0u;
  if (bit && (mask & bit)) return;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  mask |= bit;
}

int set_error(slg_ctx* ctx, int code, const char* fmt, ...);
int cuda_check(slg_ctx* ctx, cudaError_t e, const char* what);
void* scratch(slg_ctx* ctx, int slot, size_t bytes);  // nullptr on failure (error set)

// Threads that share a cell in the kernels that sum over a cell's groups.  Above
// kWarpCellGroups a block of 256 with a tree over its threads.  Up to there the
// sums have a warp's order and a warp takes a cell (eight cells per block, no
// block-wide steps) where that fills the chip, about one block per SM and 32 groups;
// with fewer cells a block forms a cell's terms and a warp adds them.  The order
// must not depend on the number of cells: a model of a batch has the values that
// it has alone.  Measured on B200, means + leakage + emission probabilities, warp /
// block: 64 cells x 512 groups 46 / 19 us, 400 x 100 21.2 / 16.6, 800 x 100 21 / 23,
// 1200 x 256 33.5 / 30.9, 2000 x 256 33.5 / 43.6, 2000 x 512 52 / 54, 16000 x 100 56 /
// 178; 8000 x 1024 239 / 255, where a block has its own order.
constexpr int kWarpCellGroups = 512;
enum CellForm { CELL_WARP, CELL_BLOCK_WARP_ORDER, CELL_BLOCK };
inline CellForm cell_form(long long cells, int ng, int num_sms) {
  if (ng > kWarpCellGroups) return CELL_BLOCK;
  return cells * 32 >= (long long)ng * num_sms ? CELL_WARP : CELL_BLOCK_WARP_ORDER;
}

// kernels launch wrappers (return SLG_OK or error)
int launch_physical_opacity(slg_ctx* ctx, const slg_gas* gas, const slg_opacity_flags* flags,
                            double* gas_sig, float* gas_cap, float* gas_emiss, double* cap64);
int launch_analytic_opacity(slg_ctx* ctx, const double* temp, const double* rho, int kind,
                            const double* coefs, double* gas_sig, float* gas_cap);
int launch_opacity_means(slg_ctx* ctx, const double* temp, const double* sig, const float* cap,
                         double* capgrey, double* capross);
int launch_leakage(slg_ctx* ctx, const double* tempinv, const double* sig, const float* cap,
                   const float* capemit, double tauddmc, double taulump, double* opaclump);
int launch_emitprob(slg_ctx* ctx, const double* tempinv, const float* cap, const double* capgrey,
                    double* emitprob);
int build_cell_tables(slg_ctx* ctx, const slg_transport_in* in);
int launch_particle_advance(slg_ctx* ctx, const slg_transport_in* in, slg_packet* prt,
                            int32_t* isvacant, int64_t npart, uint64_t seed,
                            slg_transport_out* out, uint64_t* d_trace_hash, int32_t* d_trace_nstep);
int finish_particle_advance(slg_ctx* ctx, const slg_transport_in* in, slg_transport_out* out);
int launch_fluxtally(slg_ctx* ctx, int64_t npart, const slg_packet* prt, int32_t* isvacant,
                     int flx_ng, const double* flx_wl, double* luminos, double* lumdev,
                     int32_t* lumnum);
int launch_sourcetally(slg_ctx* ctx, int64_t npart, const slg_packet* prt, const int32_t* isvacant,
                       double* src_energy, int32_t* src_number);
}  // namespace slg
