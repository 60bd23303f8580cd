// tdy_kernels.cu -- sm_103a kernels of the MPFA-O Richards residual and
// Jacobian, and their host-side launch code.
//
// One evaluation is three stages on one stream:
//   1. state_kernel   (cells, then boundary faces)
//        TDyUpdateState_Richards_MPFAO (src/fv/mpfao/tdympfao.c:2527-2594),
//        TDyMPFAO_SetBoundaryPressure + TDyMPFAOUpdateBoundaryState
//        (src/fv/mpfao/tdympfao_utils.c:24-99, 690-759) and the accumulation
//        terms of TDyMPFAOSNESFunction/Jacobian (tdympfao_snes.c:19-30,
//        112-123, 166-179) or TDyMPFAOIFunction/IJacobian_Accumulation
//        (tdympfao_ts.c:191-212, 459-517).
//   2. vertices: MatMult(Trans_mat, P_vec) (tdympfao_ts.c:184) restricted to
//        the vertex's rows, the upwinded flux of TDyMPFAOIFunction_Vertices
//        (tdympfao_ts.c:12-150) and the Jacobian entries of
//        TDyMPFAOIJacobian_Vertices (tdympfao_ts.c:235-456).  Each vertex
//        writes its partial residual R_v[nint] and partial Jacobian block
//        J_v[nint][nint] (rows and columns: the vertex's internal cells) to a
//        scratch area it alone owns.  Interior hexahedral vertices use a fixed
//        octant layout (rows and columns known at compile time, structure-of-
//        arrays storage read with coalesced loads); the others use per-vertex
//        blocks, a few lanes each, in the first blocks of the same launch.
//   3. cells: sum, in a fixed order, the partials of the cell's vertices into
//        R[cell] and into the cell's row of the fixed CSR pattern, then add
//        the accumulation terms (cell_kernel: structured cells, one thread
//        each; generic_cell_kernel: the others, a few lanes each).  No
//        atomics, and both sum in the same order: results are bitwise
//        reproducible run to run.
//
// Per row the flux is evaluated as -w*(T.P + rho_avg*G) with w = rho_avg*kr/mu
// and the Jacobian entry as -(w*T + E) with E the derivative terms of the
// up/down cell, the same quantities as the reference's
// rho*kr/mu*(-T.P) - rho^2*kr/mu*G and its five-term derivative
// (tdympfao_ts.c:116-118, 404-417) regrouped to need fewer FP64 operations.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "tdy_arena.h"
#include "tdy_device.h"
#include "tdy_emit.h"
#include "tdy_ff.h"
#include "tdy_pow.h"

namespace tdy {

#define TDY_MAX_ROWS 64
#define TDY_MAX_NINT 64
// Jacobian row length: the gather program stores slots in 8 bits
#define TDY_MAX_ROW_NNZ 255

// An other (not canonical) vertex: its rows, columns and internal cells in the
// packed arrays g_row*, g_col and g_cell, its Trans block and its partials.
struct __align__(16) GenVertex {
  long long trans, jv;
  int row0, col0, cell0;
  unsigned char nrow, ncol, nint, pad;
};

// An other (not structured) cell: where its vertices and entries start in gv_*
// and ge_*, their numbers, the diagonal's slot.
struct __align__(16) GenCellHead {
  int cell, k0, e0;
  unsigned char n, rn, diag, pad;
};

struct DevArgs {
  int nc, nb, nv;
  int form;
  int rho_type, mu_type;
  int needR, needJ;
  double Pref, dt, shift;
  // inputs
  const double *U, *Ut;
  // cells
  const double *vol, *poro, *Sr, *sat_param, *rp_param, *ss, *accum_prev;
  const double *lam_sat;  // kr(Se = 1) / mu per cell (saturated cells)
  double vis, inv_vis;    // water viscosity (constant at Tref and zero salinity) and 1 / vis
  const int *sat_type, *rp_type;
  // boundary faces
  const int *bnd_cell, *bnd_type, *bnd_has;
  const double *bnd_val, *bnd_rho, *bnd_vis;
  // extended state (cells then boundary faces): P, rho/2, (drho/dP)/2, kr/mu,
  // d(kr/mu)/dP, seepage flag
  // (constant density: lam holds rho kr/mu, every row's w)
  double *P, *hr, *hdr, *lam, *dlam;
  unsigned char *seep;
  double *acc_a, *acc_b, *jdiag;
  const double *G;  // per face
  // canonical interior-hex vertices (SoA, stride nCpad); a launch takes those in [vc0, vc1)
  int nC, nCpad, vc0, vc1;
  const double *Tc;
  // the curves by the FP64 power functions only: the device Newton's iteration
  // counts at the rounding floor follow the last bits of the residual, and
  // stay what they were
  int fp64_curves;
  int jac_ff;  // Jacobian products of canonical vertices in double-float
  const int *cellc, *facec;
  // other vertices: gen_lanes threads each, gen_doubles of shared memory
  int ngen, gen_lanes, gen_apart, gen_doubles, gen_max_row, gen_max_col;
  const GenVertex *gen;
  const int *g_col;      // extended index of a column
  const double *g_rowG;  // gravity coefficient of a row
  const uchar2 *g_rowc;  // columns of a row's up and down sides
  const uint2 *g_cell;   // of an internal cell: see gen_cell_program
  const double *trans;
  double *scratch;
  // cell gather
  const int *rowptr;
  const GenCellHead *gc;
  const long long *gv_j, *gv_r;
  const unsigned long long *ge_code;
  const unsigned *gv_n;
  const unsigned char *ge_slot;
  int ge_words, gc_max_vals;
  int max_row_nnz;
  // instances: of each cell, and (a call on some instances only, else null)
  // which are evaluated; the others' entities are skipped
  const int *cell_inst, *inst_on;
  int nS, nSpad, ngc;
  const int *sc_cells, *sc_vc;
  // outputs
  double *R, *J;
};

// whether the instance of a cell is evaluated
__device__ __forceinline__ bool inst_skipped(const DevArgs &a, int cell) {
  return a.inst_on && !a.inst_on[a.cell_inst[cell]];
}

// timer groups: the state kernel, the vertex kernels, the cell kernels
static const char *const kKernelNames[3] = {"state_kernel", "vertex_kernel", "cell_kernel"};

struct DeviceState {
  cudaStream_t stream = nullptr;
  DevArgs a;
  // per-kernel timers (TDY_START_FUNCTION_TIMER analogue, include/tdytimers.h)
  bool timers = false;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  double t_ms[3] = {0, 0, 0};
  long long t_calls[3] = {0, 0, 0};
  int device = 0;  // CUDA device current at TDySetup
  // owned allocations
  std::vector<void *> allocs;
  double *dU = nullptr, *dUt = nullptr, *dR = nullptr, *dJ = nullptr;
  double *diagS = nullptr, *diagMass = nullptr;
  double *dae = nullptr;  // DAE form: U, U_t, R interleaved (6 * nc), on first use
  int nnz = 0;
  // host-pointer evaluations in slabs of cells (see build_slabs): each slab's
  // rows of R and J go to host memory while the next slabs are evaluated
  struct Slab {
    int e0, e1;        // cells whose state this slab computes (its vertices read up to e1)
    int c0, c1;        // cells
    int vc0, vc1;      // canonical vertices
    int g0, g1;        // other vertices (indices into gen_vertex)
    int s0, s1;        // structured cells (indices into sc_cells)
    int gc0, gc1;      // other cells (indices into gc_cells)
    long long j0, j1;  // Jacobian values
  };
  std::vector<Slab> slabs;
  cudaStream_t copy_stream = nullptr;
  std::vector<cudaEvent_t> slab_ev;
  // the slab pipeline as one graph for pinned host buffers, with what its
  // nodes bake in (rebuilt when a call differs)
  struct SlabKey {
    int form = -1;
    double dt = 0.0, shift = 0.0;
    const double *U = nullptr, *Ut = nullptr;
    double *R = nullptr, *J = nullptr;
    bool operator==(const SlabKey &o) const {
      return form == o.form && dt == o.dt && shift == o.shift && U == o.U && Ut == o.Ut && R == o.R && J == o.J;
    }
  };
  cudaGraphExec_t slab_exec = nullptr;
  SlabKey slab_key;
  // callers' streams that enqueued work on this handle, each with an event
  // recorded after its last enqueue: TDyDestroy waits for them before the
  // stream-ordered frees (which do not synchronise the device)
  std::vector<std::pair<cudaStream_t, cudaEvent_t>> user_streams;
  // calls on some instances: their flags on the device, and the host's copy
  int *inst_on = nullptr;
  std::vector<int> h_on;
  bool inst_ok = false;
  // recorded after every allocation-free evaluation (created at set-up, so
  // that call creates nothing); such calls never overlap, so the last one
  // covers them all
  cudaEvent_t noalloc_ev = nullptr;
};

#define CUDA_TRY(call)                                                                          \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      return set_error(TDY_ERR_GPU, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

// ---------------------------------------------------------------------------
// Constitutive relations, restated from src/materials/tdycharacteristiccurves.c
// and src/materials/tdyeos.c with the reference's operation order.

// PressureSaturation_VanGenuchten (tdycharacteristiccurves.c:692-717) and
// PressureSaturation_Gardner (:641-667).
__device__ __forceinline__ void saturation(int type, const double *par, double Sr, double Pc, double *S, double *dS,
                                           double *d2S) {
  if (type == SAT_FUNC_VAN_GENUCHTEN) {
    const double m = par[0], alpha = par[1];
    if (Pc <= 0) {
      *S = 1;
      *dS = 0;
      *d2S = 0.0;
    } else {
      // PressureSaturation_VanGenuchten (tdycharacteristiccurves.c:692-717)
      // with two powers instead of four: (1 + x^n)^(m+1) = (1 + x^n) / Se and
      // (1 + x^n)^(-m-2) = Se / (1 + x^n)^2 (FP64 pow is the cost here)
      double n = 1 / (1 - m);
      double pc_alpha = Pc * alpha;
      double pc_alpha_n = pow(pc_alpha, n);
      double one_plus = 1 + pc_alpha_n;
      double Se = pow(one_plus, -m);
      *S = (1.0 - Sr) * Se + Sr;
      double dSe_dPc = -m * n * alpha * pc_alpha_n * Se / (pc_alpha * one_plus);
      *dS = -dSe_dPc * (1.0 - Sr);
      double d2Se = m * n * pc_alpha_n * (Se / (one_plus * one_plus)) * ((m * n + 1.0) * pc_alpha_n - n + 1) / (Pc * Pc);
      *d2S = (1.0 - Sr) * d2Se;
    }
  } else {
    const double m = par[1], alpha = par[2];
    if (Pc < 0) {
      *S = 1;
      *dS = 0;
      *d2S = 0.0;
    } else {
      double Se = exp(-alpha * Pc / m);
      *S = (1.0 - Sr) * Se + Sr;
      double dSe_dPc = -alpha / m * exp(-alpha * Pc / m);
      *dS = -dSe_dPc * (1.0 - Sr);
      double d2Se = -alpha / m * dSe_dPc;
      *d2S = (1.0 - Sr) * d2Se;
    }
  }
}

// RelativePermeability_Mualem (tdycharacteristiccurves.c:468-485, 551-562,
// 607-614) and RelativePermeability_Irmay (:451-460).
__device__ __forceinline__ void relperm(int type, const double *p, double Se, double *Kr, double *dKr) {
  if (type == REL_PERM_FUNC_MUALEM) {
    const double m = p[0], x0 = p[1], x1 = p[2], dx = p[4];
    if (Se > x1) {
      double xt = (Se - x0) / dx;
      *Kr = p[5] + xt * (p[6] + xt * (p[7] + xt * p[8]));
      *dKr = (p[6] + xt * (2.0 * p[7] + xt * 3.0 * p[8])) / dx;
    } else {
      *Kr = 1.0;
      *dKr = 0.0;
      if (Se >= 1.0) return;
      // two powers instead of five: Se^(1/m - 1/2) = so / sqrt(Se),
      // (1 - so)^(m-1) = tmp / (1 - so), (1 - so)^m = tmp
      double so = pow(Se, 1 / m);
      double oms = 1 - so;
      double tmp = pow(oms, m);
      double sq = sqrt(Se);
      double kr = sq * ((1 - tmp) * (1 - tmp));
      *Kr = kr;
      double d = 0.5 * kr / Se;
      d += 2 * (so / sq) * (tmp / oms) * (1 - tmp);
      *dKr = d;
    }
  } else {
    const double m = p[0];
    *Kr = 1.0;
    *dKr = 0.0;
    if (Se >= 1.0) return;
    *Kr = pow(Se, m);
    *dKr = pow(Se, m - 1) * m;
  }
}

// EOSComputeWaterDensity / EOSComputeWaterViscosity (tdyeos.c:5-136) at
// T = Tref and zero salinity.
// EOSComputeWaterDensity_Constant (tdyeos.c:5-14)
constexpr double kRhoConst = 998.0;

__device__ __forceinline__ void density(int type, double p, double *rho, double *drho, double *d2rho) {
  if (type == WATER_DENSITY_CONSTANT) {
    *rho = kRhoConst;
    *drho = 0.0;
    *d2rho = 0.0;
  } else if (type == WATER_DENSITY_EXPONENTIAL) {
    if (p < 101325.e0) {
      *rho = 997.16e0;
      *drho = 0.0;
      *d2rho = 0.0;
    } else {
      double r = 997.16e0 * exp(1.e-8 * (p - 101325.e0));
      *rho = r;
      *drho = 1.e-8 * r;
      *d2rho = 1.e-8 * (1.e-8 * r);
    }
  } else {
    const double T = 25.0, P = p * 1.e-6;
    double pw = 1 + 1.e-6 * (-80. * T - 3.3 * (T * T) + 0.00175 * (T * T * T) + 489. * P - 2. * T * P +
                             0.016 * P * (T * T) - 1.3e-5 * (T * T * T) * P - 0.333 * (P * P) - 0.002 * T * (P * P));
    *rho = pw * 1000.;
    *drho = 0.0;
    *d2rho = 0.0;
  }
}

__device__ __forceinline__ void viscosity(int type, double *vis, double *dvis) {
  if (type == WATER_VISCOSITY_CONSTANT) {
    *vis = 9.94e-4;
  } else {
    const double T = 25.0;
    *vis = (0.1 + 1.65 * exp((-0.42 * (0.17 * 0.17) + 0.045) * pow(T, 0.8))) * 1e-3;
  }
  *dvis = 0.0;
}

// Saturation and mobility of an unsaturated cell: S, dS/dP, d2S/dP2, kr and
// dkr/dP.
struct Curves {
  double S, dS, d2S, kr, dkr;
};

// van Genuchten saturation with Mualem relative permeability of the same m,
// by the identities of their bases: with x = alpha Pc and w = 1 + x^n,
//   Se = w^-m,  Se^(1/m) = 1/w,  (1 - Se^(1/m))^m = (x^n / w)^m =: t,
// so kr = sqrt(Se) (1 - t)^2 and, with x^(nm) = x^(n-1),
//   -dSe/dPc = m n alpha x^(n-1) Se / w,
//   dkr/dSe = kr / (2 Se) + 2 sqrt(Se) (1 - t) / x.
// Every power comes from log2 x and log2 w by one exp2_fx (tdy_pow.h): in FP64
// the four powers and eleven divisions of the plain formulas took a warp 33 k
// cycles (one cell per lane); the state stage of 204 k unsaturated cells took
// 0.225 ms and takes 0.035 ms so.
// The cell's parameters: par = m, alpha, n; p = the Mualem parameters.  False
// (nothing set) outside the range of the integer powers, whose exponents are
// positive: m above 1 makes n negative.
__device__ __forceinline__ bool vg_mualem(const double *par, const double *p, double Sr, double Pc, bool want_kr,
                                          bool want_d, bool want_d2, Curves *c) {
  const double m = par[0], alpha = par[1], n = par[2];
  const double x = __dmul_rn(Pc, alpha);
  const int be = (int)((unsigned)__double2hiint(x) >> 20) - 1023;  // (a set sign bit puts it out of range)
  if (!(be > -300 && be < 300 && m >= 0.00390625 && n >= 1.0 && n <= 32.0 && (abs(be) + 1) * (int)(n + 1.0) < 500)) return false;
  const fx lx = log2_fx(x), tn = fx_scale(n, lx);
  const double xn = exp2_fx(tn), w = __dadd_rn(1.0, xn);
  const fx lw = log2_fx(w), mw = fx_scale(m, lw);
  const double Se = exp2_fx(fx_neg(mw)), oms = __dadd_rn(1.0, -Sr);
  c->S = __fma_rn(oms, Se, Sr);
  if (!want_kr && !want_d) return true;
  double g = 0.0, u = 0.0, xi = 0.0, us = 0.0;  // us: x^(n-1) Se
  if (want_d) {
    const double wi = exp2_fx(fx_neg(lw)), mn = __dmul_rn(m, n);
    xi = exp2_fx(fx_neg(lx));
    u = __dmul_rn(xn, xi);
    g = __dmul_rn(__dmul_rn(mn, alpha), wi);
    us = __dmul_rn(u, Se);
    c->dS = __dmul_rn(__dmul_rn(g, us), oms);
    if (want_d2) {
      const double q = __dmul_rn(__dmul_rn(mn, __dmul_rn(__dmul_rn(u, xi), __dmul_rn(alpha, alpha))), __dmul_rn(Se, __dmul_rn(wi, wi)));
      c->d2S = __dmul_rn(__dmul_rn(oms, q), __dadd_rn(__fma_rn(__dadd_rn(mn, 1.0), xn, -n), 1.0));
    }
  }
  if (!want_kr) return true;
  if (Se > p[2]) {  // the smoothing cubic (tdycharacteristiccurves.c:607-614)
    const double dx = p[4], xt = (Se - p[1]) / dx;
    c->kr = p[5] + xt * (p[6] + xt * (p[7] + xt * p[8]));
    if (want_d) c->dkr = __dmul_rn((p[6] + xt * (2.0 * p[7] + xt * 3.0 * p[8])) / dx, __dmul_rn(g, us));
    return true;
  }
  // f = 1 - t cancels in dry soil, where s = 1/w is small: there by the
  // binomial series of 1 - (1 - s)^m (its sixth term is below 2^-47), else
  // before any rounding.  kr is then within 1e-13 of 300-bit arithmetic (x
  // 0.03 to 1e6, m 0.2 to 0.6: 7.8e-14); the plain formulas are 2.5e-11 off up
  // to x = 100, 1.3e-6 up to 1e4 and 0.07 up to 1e6.
  double f;
  if (lw.k >= 9) {
    const double so = exp2_fx(fx_neg(lw));
    f = __fma_rn(__dmul_rn(__dadd_rn(4.0, -m), 0.2), so, 1.0);
    f = __fma_rn(__dmul_rn(__dmul_rn(__dadd_rn(3.0, -m), 0.25), so), f, 1.0);
    f = __fma_rn(__dmul_rn(__dmul_rn(__dadd_rn(2.0, -m), 1.0 / 3.0), so), f, 1.0);
    f = __fma_rn(__dmul_rn(__dmul_rn(__dadd_rn(1.0, -m), 0.5), so), f, 1.0);
    f = __dmul_rn(__dmul_rn(m, so), f);
  } else {
    f = one_minus_exp2_fx(fx_scale(m, fx_add(tn, fx_neg(lw))));
  }
  const double sq = exp2_fx(fx_neg(fx_half(mw)));
  c->kr = __dmul_rn(sq, __dmul_rn(f, f));
  if (want_d)
    c->dkr = __dmul_rn(g, __fma_rn(__dmul_rn(0.5, c->kr), u, __dmul_rn(__dmul_rn(2.0, __dmul_rn(sq, xi)), __dmul_rn(f, us))));
  return true;
}

// any curves, in FP64 (out of line: few cells take it, and inlined its powers
// would set the registers of every kernel)
__device__ __noinline__ void curves_general(int sat_type, const double *par, int rp_type, const double *p, double Sr,
                                            double Pc, Curves *c) {
  saturation(sat_type, par, Sr, Pc, &c->S, &c->dS, &c->d2S);
  const double Se = (c->S - Sr) / (1.0 - Sr);
  double dKr_dSe;
  relperm(rp_type, p, Se, &c->kr, &dKr_dSe);
  const double dSe_dS = 1.0 / (1.0 - Sr);
  c->dkr = dKr_dSe * dSe_dS * c->dS;
}

__device__ __forceinline__ Curves curves_at(const DevArgs &a, int cell, double Pc, bool want_kr, bool want_d,
                                            bool want_d2) {
  Curves c = {0.0, 0.0, 0.0, 0.0, 0.0};
  const double *par = a.sat_param + 3 * (size_t)cell, *p = a.rp_param + 9 * (size_t)cell;
  const int st = a.sat_type[cell], rt = a.rp_type[cell];
  const double Sr = a.Sr[cell];
  if (!(!a.fp64_curves && st == SAT_FUNC_VAN_GENUCHTEN && Pc > 0 && (!want_kr || (rt == REL_PERM_FUNC_MUALEM && p[0] == par[0])) &&
        vg_mualem(par, p, Sr, Pc, want_kr, want_d, want_d2, &c)))
    curves_general(st, par, rt, p, Sr, Pc, &c);
  return c;
}

// van Genuchten Pc <= 0, Gardner Pc < 0: S = 1, dS = 0
__device__ __forceinline__ bool saturated_at(int sat_type, double Pc) {
  return (sat_type == SAT_FUNC_VAN_GENUCHTEN) ? (Pc <= 0) : (Pc < 0);
}

// S and, with want_d, dS/dP of any cell
__device__ __forceinline__ Curves cell_saturation(const DevArgs &a, int cell, double Pc, bool want_d) {
  if (saturated_at(a.sat_type[cell], Pc)) return Curves{1.0, 0.0, 0.0, 0.0, 0.0};
  return curves_at(a, cell, Pc, false, want_d, false);
}

// x / vis, correctly rounded but for rare ties, without the FP64 division
__device__ __forceinline__ double over_vis(const DevArgs &a, double x) {
  if (a.fp64_curves) return x / a.vis;
  const double q = __dmul_rn(x, a.inv_vis);
  return __fma_rn(__fma_rn(-q, a.vis, x), a.inv_vis, q);
}

// ---------------------------------------------------------------------------
// 1. cell and boundary-face state
// Warps take 32-entity chunks in the order chunk = (warp * chunk_mul) mod
// nchunks (chunk_mul coprime to nchunks): loads stay coalesced within a warp
// while the unsaturated cells, which cost ~10x more and cluster in space
// (and therefore in cell numbering), spread over every SM instead of forming
// a tail of a few slow blocks.
// entity i: cell i < nc, else boundary face i - nc
__device__ __forceinline__ void state_entity(const DevArgs &a, int i) {
  if (i < a.nc) {
    if (inst_skipped(a, i)) return;
    const double U = a.U[i];
    const double Pc = a.Pref - U;
    const double P = a.Pref - Pc;
    // Saturated cells: Se = (1 - Sr)/(1 - Sr) = 1 exactly, so kr/mu is the
    // per-cell constant lam_sat and its pressure derivative is zero.
    double S = 1.0, dS = 0.0, d2S = 0.0, lam, dlam = 0.0;
    const bool saturated = saturated_at(a.sat_type[i], Pc);
    if (saturated) {
      lam = a.lam_sat[i];
    } else {
      const Curves c = curves_at(a, i, Pc, true, a.needJ || a.form == FORM_TS, a.form == FORM_TS && a.needJ);
      S = c.S;
      dS = c.dS;
      d2S = c.d2S;
      lam = over_vis(a, c.kr);
      dlam = over_vis(a, c.dkr);  // the viscosity does not depend on pressure here
    }
    double rho, drho, d2rho;
    density(a.rho_type, P, &rho, &drho, &d2rho);
    a.P[i] = P;
    if (a.rho_type != WATER_DENSITY_CONSTANT) {  // (constant: no vertex gathers it)
      a.hr[i] = 0.5 * rho;
      a.hdr[i] = 0.5 * drho;
    }
    a.lam[i] = a.rho_type == WATER_DENSITY_CONSTANT ? __dmul_rn(kRhoConst, lam) : lam;
    a.dlam[i] = dlam;
    const double poro = a.poro[i], vol = a.vol[i];
    // d(rho phi S)/dP (the porosity does not depend on pressure)
    double dmass = rho * poro * dS;
    if (a.rho_type != WATER_DENSITY_CONSTANT) dmass = drho * poro * S + rho * poro * dS;
    if (a.form == FORM_SNES) {
      const double dtInv = a.shift;  // 1/dt, computed on the host
      double acc = rho * poro * S * vol * dtInv;
      a.acc_a[i] = acc - a.accum_prev[i];
      a.acc_b[i] = a.ss[i];
      a.jdiag[i] = saturated && a.rho_type == WATER_DENSITY_CONSTANT ? 0.0 : dmass * vol * dtInv;
    } else if (a.form == FORM_TV) {
      // TDyMPFAOIFunction_TransientVariable (tdympfao_ts_transientvar.c:89-95):
      // Ut holds dM/dt; the Jacobian adds shift * dM/dP * V.
      a.acc_a[i] = a.Ut[i] * vol;
      a.acc_b[i] = a.ss[i] * vol;
      a.jdiag[i] = a.shift * dmass * vol;
    } else {
      const double Ut = a.Ut[i];
      // d2(rho phi S)/dP2 with constant porosity
      const double d2mass = (S * d2rho + 2.0 * (dS * drho) + d2S * rho) * poro;
      a.acc_a[i] = dmass * Ut * vol;
      a.acc_b[i] = a.ss[i] * vol;
      a.jdiag[i] = (a.shift * dmass + d2mass * Ut) * vol;
    }
  } else if (i < a.nc + a.nb) {
    const int b = i - a.nc;
    if (a.bnd_type[b] == NEUMANN_BC) return;  // no vertex row or column uses it
    const int c = a.bnd_cell[b];
    if (inst_skipped(a, c)) return;
    const double p = a.bnd_has[b] ? a.bnd_val[b] : a.U[c];
    const double Pc = a.Pref - p;
    double lam;
    if (saturated_at(a.sat_type[c], Pc)) {
      lam = a.lam_sat[c];  // kr(1) / mu with the boundary viscosity (the same constant)
    } else {
      const Curves cv = curves_at(a, c, Pc, true, false, false);
      lam = cv.kr / a.bnd_vis[b];
    }
    a.P[i] = p;
    if (a.rho_type != WATER_DENSITY_CONSTANT) {
      a.hr[i] = 0.5 * a.bnd_rho[b];
      a.hdr[i] = 0.0;
    }
    a.lam[i] = a.rho_type == WATER_DENSITY_CONSTANT ? __dmul_rn(kRhoConst, lam) : lam;
    a.dlam[i] = 0.0;
    a.seep[i] = (a.bnd_type[b] == SEEPAGE_BC && p <= a.Pref) ? 1 : 0;
  }
}

// entities [e0, e1) (cells below nc, then boundary faces)
__global__ void __launch_bounds__(256) state_kernel(DevArgs a, int e0, int e1, int nchunks, int chunk_mul) {
  const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (gw >= nchunks) return;
  const int i = e0 + (int)(((long long)gw * chunk_mul) % nchunks) * 32 + (int)(threadIdx.x & 31);
  if (i < e1) state_entity(a, i);
}

// Accumulation at the previous solution (TDyMPFAOSNESPreSolve,
// tdympfao_snes.c:19-64).
__global__ void __launch_bounds__(256) presolve_kernel(DevArgs a, const double *Uprev, double *accum_prev) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nc) return;
  const double Pc = a.Pref - Uprev[i];
  const double S = cell_saturation(a, i, Pc, false).S;
  double rho, drho, d2rho;
  density(a.rho_type, a.Pref - Pc, &rho, &drho, &d2rho);
  accum_prev[i] = rho * a.poro[i] * S * a.vol[i] / a.dt;
}

// Transient variable (TDyMPFAOTransientVariable, tdympfao_ts_transientvar.c:
// 13-47): C = rho phi S V, and its pressure derivative.
__global__ void __launch_bounds__(256) tv_kernel(DevArgs a, const double *U, double *C, double *dC) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nc) return;
  const double Pc = a.Pref - U[i];
  const Curves c = cell_saturation(a, i, Pc, dC != nullptr);
  double rho, drho, d2rho;
  density(a.rho_type, a.Pref - Pc, &rho, &drho, &d2rho);
  const double poro = a.poro[i], vol = a.vol[i];
  if (C) C[i] = rho * poro * c.S * vol;
  if (dC) dC[i] = (drho * poro * c.S + rho * poro * c.dS) * vol;
}

// DAE form (TDyMPFAOIFunction_DAE, tdympfao_ts_dae.c:13-84): split the
// interleaved [P, M] unknowns, then combine R_P (the transient-variable
// residual with dM/dt) and R_M = M - rho phi S V.
__global__ void __launch_bounds__(256) dae_split_kernel(int n, const double *U2, const double *Ut2, double *P,
                                                        double *Mdot) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  P[i] = U2[2 * i];
  Mdot[i] = Ut2[2 * i + 1];
}
__global__ void __launch_bounds__(256) dae_merge_kernel(int n, const double *U2, const double *Rp, const double *C,
                                                        double *R2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  R2[2 * i] = Rp[i];
  R2[2 * i + 1] = U2[2 * i + 1] - C[i];
}

// Diagnostics (TDyUpdateDiagnostics_MPFAO, tdympfao.c:2780-2806): saturation
// and rho*V per cell.
__global__ void __launch_bounds__(256) diag_kernel(DevArgs a, double *Sout, double *mass) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nc) return;
  const double Pc = a.Pref - a.U[i];
  const double S = cell_saturation(a, i, Pc, false).S;
  double rho, drho, d2rho;
  density(a.rho_type, a.Pref - Pc, &rho, &drho, &d2rho);
  Sout[i] = S;
  mass[i] = rho * a.vol[i];
}

// ---------------------------------------------------------------------------
// 2. interior hexahedral vertices, octant layout

// Octants joined by canonical row r (kCanonUp/kCanonDn in tdy_internal.h).
__host__ __device__ constexpr int canon_up(int r) {
  return r < 4 ? 2 * r : r < 8 ? (((r - 4) & 1) | (((r - 4) >> 1) << 2)) : r - 8;
}
__host__ __device__ constexpr int canon_dn(int r) { return canon_up(r) | (1 << (r / 4)); }
static_assert(canon_up(5) == kCanonUp[5] && canon_dn(5) == kCanonDn[5] && canon_up(10) == kCanonUp[10] &&
                  canon_dn(10) == kCanonDn[10] && canon_up(2) == kCanonUp[2] && canon_dn(7) == kCanonDn[7],
              "canonical row tables disagree");

// Corner offsets, octants and slots of structured cells (kCornerOffset,
// struct_octant, struct_slot in tdy_internal.h) without host tables.
__host__ __device__ constexpr int corner_offset(int j) { return j ^ ((j >> 1) & 1); }
__host__ __device__ constexpr int d_struct_octant(int j) { return 7 ^ corner_offset(j); }
__host__ __device__ constexpr int d_struct_slot(int j, int b) {
  return ((((corner_offset(j) >> 2) & 1) - 1 + ((b >> 2) & 1)) + 1) * 9 +
         ((((corner_offset(j) >> 1) & 1) - 1 + ((b >> 1) & 1)) + 1) * 3 + (((corner_offset(j) & 1) - 1 + (b & 1)) + 1);
}
// whether corner j is the first of a structured cell's corners whose vertex
// touches octant b's slot
__host__ __device__ constexpr bool first_touch(int j, int b) {
  for (int i = 0; i < j; i++)
    for (int o = 0; o < 8; o++)
      if (d_struct_slot(i, o) == d_struct_slot(j, b)) return false;
  return true;
}
static_assert(corner_offset(2) == kCornerOffset[2] && corner_offset(7) == kCornerOffset[7] &&
                  d_struct_slot(0, 7) == struct_slot(0, 7) && d_struct_slot(6, 0) == struct_slot(6, 0) &&
                  d_struct_slot(3, 5) == struct_slot(3, 5),
              "structured-cell tables disagree");

// Row of the canonical layout that joins octant c with its neighbour across
// axis k, and whether c is that row's first ("up") cell.
__host__ __device__ constexpr int canon_row(int c, int k) {
  return k == 0 ? ((c & ~1) >> 1) : k == 1 ? 4 + (((c & ~2) & 1) | (((c & ~2) >> 2) << 1)) : 8 + (c & ~4);
}
__host__ __device__ constexpr bool canon_is_up(int c, int k) { return ((c >> k) & 1) == 0; }

// x < 0.0 by integer operations (the FP64 pipe is this kernel's bound):
// the sign bit set, and neither a zero nor a NaN
__device__ __forceinline__ bool dneg(double x) {
  const long long b = __double_as_longlong(x), m = b & 0x7fffffffffffffffLL;
  return b < 0 && m != 0 && m <= 0x7ff0000000000000LL;
}

// first canonical row that touches octant o
__host__ __device__ constexpr int canon_first_row(int o) {
  for (int r = 0; r < 12; r++)
    if (canon_up(r) == o || canon_dn(r) == o) return r;
  return -1;
}

// Density modes of the canonical vertex: RHO_CONST (constant density: the
// face average 2 (rho/2) is the constant itself, rho/2 is not gathered),
// RHO_NODERIV (density without a pressure derivative), RHO_EXP (exponential,
// with its derivative).
enum { RHO_CONST = 0, RHO_NODERIV = 1, RHO_EXP = 2 };

// canonical vertex vc with FP64 Jacobian products; tid: its slot of the
// block's shared rows
template <int RHO>
__device__ __forceinline__ void canon_vertex_at(const DevArgs &a, int vc, int tid) {
  constexpr bool CONST_RHO = RHO != RHO_EXP;
  extern __shared__ double sh[];  // [36][blockDim]: w, E_up, E_dn per row
  const int bs = blockDim.x;
  const long long P = a.nCpad;
  double p[8], hr[8], lam[8], dlam[8], hdr[8];
#pragma unroll
  for (int o = 0; o < 8; o++) {
    const int cell = a.cellc[o * P + vc];
    p[o] = a.P[cell];
    hr[o] = RHO == RHO_CONST ? 0.5 * kRhoConst : a.hr[cell];
    lam[o] = a.lam[cell];
    dlam[o] = a.dlam[cell];
    hdr[o] = CONST_RHO ? 0.0 : a.hdr[cell];
  }
  double Rv[8];
#pragma unroll
  for (int r = 0; r < 12; r++) {
    const int u = canon_up(r), d = canon_dn(r);
    const double *T = a.Tc + (long long)(r * 8) * P + vc;
    // explicit roundings: the same bits whichever outputs a call requests
    double TP = __dmul_rn(T[0], p[0]);
#pragma unroll
    for (int c = 1; c < 8; c++) TP = __fma_rn(T[c * P], p[c], TP);
    const double G = a.G[a.facec[r * P + vc]];
    // (constant density: 499 + 499, exactly the constant)
    const double den = RHO == RHO_CONST ? kRhoConst : __dadd_rn(hr[u], hr[d]);
    const double q = __fma_rn(den, G, TP);
    const bool fdn = dneg(q);
    const double lm = fdn ? lam[u] : lam[d];
    const double w = RHO == RHO_CONST ? lm : __dmul_rn(den, lm);
    const double flux = -__dmul_rn(w, q);
    // an octant's partial residual starts from its first row's flux
    if (r == canon_first_row(u))
      Rv[u] = flux;
    else
      Rv[u] += flux;
    if (r == canon_first_row(d))
      Rv[d] = -flux;
    else
      Rv[d] -= flux;
    if (a.needJ) {
      // derivative of the flux with respect to the up and down cell pressures
      // beyond w*T: d(rho_avg)/dP and d(kr/mu)/dP of the upwind cell
      double eu, ed;
      if (CONST_RHO) {
        const double e = __dmul_rn(__dmul_rn(den, q), fdn ? dlam[u] : dlam[d]);
        eu = fdn ? e : 0.0;
        ed = fdn ? 0.0 : e;
      } else {
        const double dlu = fdn ? dlam[u] : 0.0, dld = fdn ? 0.0 : dlam[d];
        const double g2 = __fma_rn(den, G, q);
        eu = __fma_rn(__dmul_rn(hdr[u], lm), g2, __dmul_rn(__dmul_rn(den, dlu), q));
        ed = __fma_rn(__dmul_rn(hdr[d], lm), g2, __dmul_rn(__dmul_rn(den, dld), q));
      }
      sh[r * bs + tid] = w;
      sh[(12 + r) * bs + tid] = eu;
      sh[(24 + r) * bs + tid] = ed;
    }
  }
  double *S = a.scratch;
  if (a.needR) {
#pragma unroll
    for (int c = 0; c < 8; c++) S[64 * P + c * P + vc] = Rv[c];
  }
  if (!a.needJ) return;
  // J_v[c][b] = sum over the three rows k of octant c of
  //   -+ w_r T_rb  (minus when c is the row's up cell)  -+ E terms
#pragma unroll
  for (int c = 0; c < 8; c++) {
    double out[8];
#pragma unroll
    for (int b = 0; b < 8; b++) out[b] = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int r = canon_row(c, k);
      const bool up = canon_is_up(c, k);
      const double wr = sh[r * bs + tid];
      const double sw = up ? -wr : wr;
      const double *T = a.Tc + (long long)(r * 8) * P + vc;
#pragma unroll
      for (int b = 0; b < 8; b++) out[b] = __fma_rn(sw, T[b * P], out[b]);
      const double eu = sh[(12 + r) * bs + tid], ed = sh[(24 + r) * bs + tid];
      const int u = canon_up(r), d = canon_dn(r);
      out[u] = __dadd_rn(out[u], up ? -eu : eu);
      out[d] = __dadd_rn(out[d], up ? -ed : ed);
    }
    // J_v[c][0..7] is 64 contiguous bytes at [c][vc][b]
    double2 *dst = reinterpret_cast<double2 *>(S + ((long long)c * P + vc) * 8);
    dst[0] = make_double2(out[0], out[1]);
    dst[1] = make_double2(out[2], out[3]);
    dst[2] = make_double2(out[4], out[5]);
    dst[3] = make_double2(out[6], out[7]);
  }
}

// Canonical vertex vc by a lane pair (h = lane parity; slot: the pair's
// column of the block's ns shared rows), double-float Jacobian products.
// Lane h computes rows 2h+i (x), 4+2h+i (y) and 8+2h+i (z), i = 0, 1: the x
// and y rows of octants 4h..4h+3 and half of their z rows (the other half
// comes from the partner by a shuffle); it writes R_v of octants 4h..4h+3 and
// entries 4h..4h+3 (relative to the octant, column j ^ c) of every octant's
// J_v.  Rows, fluxes and R_v are formed by the operations of canon_vertex_at in
// the same order (the same bits).  A pair holds half the live state of one
// thread (the upwind cell data sit in shared memory), which doubles the warps
// that hide the FP64 latency.  J_v's octants go in a runtime loop (small enough
// for the instruction cache), entries indexed relative to the octant, j = b ^ c,
// so that the row of axis k touches entries 0 (c itself) and 1 << k at
// compile-time register indices.  Each entry is accumulated at its own
// power-of-two scale, chosen from the exponent fields of its terms so that its
// largest term is O(1): entries of rows upwinded from nearly dry cells (kr ~
// 1e-30 and below) keep full relative accuracy next to O(1) entries.
constexpr int pair_shared_rows(int rho) { return 36 + 16 + (rho == 0 ? 0 : 8) + (rho == 2 ? 8 : 0); }
// (warp, for the constant density: the lanes of the warp that call it)
template <int RHO>
__device__ __forceinline__ void canon_vertex_pair(const DevArgs &a, int vc, int slot, int h, int ns, unsigned warp) {
  constexpr bool CONST_RHO = RHO != RHO_EXP;
  // [36][ns]: w, E_up, E_dn per row; [8][ns] kr/mu and d(kr/mu)/dP per
  // octant; rho/2 and d(rho/2)/dP per octant where the density varies
  extern __shared__ double sh[];
  double *s_lam = sh + 36 * ns, *s_dlam = s_lam + 8 * ns, *s_hr = s_dlam + 8 * ns, *s_hdr = s_hr + 8 * ns;
  const unsigned pm = 3u << ((threadIdx.x & 31) & ~1);
  const long long P = a.nCpad;
  double p[8];
#pragma unroll
  for (int o = 0; o < 8; o++) {
    const int cell = a.cellc[o * P + vc];
    p[o] = a.P[cell];
    if ((o >> 2) == h) {
      s_lam[o * ns + slot] = a.lam[cell];
      s_dlam[o * ns + slot] = a.dlam[cell];
      if (RHO != RHO_CONST) s_hr[o * ns + slot] = a.hr[cell];
      if (!CONST_RHO) s_hdr[o * ns + slot] = a.hdr[cell];
    }
  }
  __syncwarp(pm);
  double fx[2], fy[2], fz[2];
  // octant of the up side of the lane's row t (canon_up)
  auto up_octant = [&](int axis, int i) { return h ? (axis == 0 ? 4 + 2 * i : axis == 1 ? 4 + i : 2 + i) : (axis == 0 ? 2 * i : i); };
  unsigned down = 0;  // constant density: bit t, the row's upwind cell is its up cell
  long long any_e = 0;
#pragma unroll
  for (int t = 0; t < 6; t++) {
    const int axis = t >> 1, i = t & 1;
    const int r = 4 * axis + 2 * h + i;
    const int u = up_octant(axis, i);
    const int d = u + (1 << axis);
    const double *T = a.Tc + (long long)(r * 8) * P + vc;
    double TP = __dmul_rn(T[0], p[0]);
#pragma unroll
    for (int c = 1; c < 8; c++) TP = __fma_rn(T[c * P], p[c], TP);
    const double G = a.G[a.facec[r * P + vc]];
    const double den = RHO == RHO_CONST ? kRhoConst : __dadd_rn(s_hr[u * ns + slot], s_hr[d * ns + slot]);
    const double q = __fma_rn(den, G, TP);
    const bool fdn = dneg(q);
    const int uw = fdn ? u : d;  // upwind octant
    const double lm = s_lam[uw * ns + slot];
    const double w = RHO == RHO_CONST ? lm : __dmul_rn(den, lm);
    const double flux = -__dmul_rn(w, q);
    (axis == 0 ? fx : axis == 1 ? fy : fz)[i] = flux;
    if (a.needJ) {
      const double dl = s_dlam[uw * ns + slot];
      double eu, ed;
      if (RHO == RHO_CONST) {
        // E below, for the warps that have any (dl = 0 in saturated cells)
        eu = q;
        ed = 0.0;
        down |= (unsigned)fdn << t;
        any_e |= __double_as_longlong(dl) << 1;
        any_e |= d_bexp(q) == 0x7ff;
      } else if (CONST_RHO) {
        const double e = __dmul_rn(__dmul_rn(den, q), dl);
        eu = fdn ? e : 0.0;
        ed = fdn ? 0.0 : e;
      } else {
        const double dlu = fdn ? dl : 0.0, dld = fdn ? 0.0 : dl;
        const double g2 = __fma_rn(den, G, q);
        eu = __fma_rn(__dmul_rn(s_hdr[u * ns + slot], lm), g2, __dmul_rn(__dmul_rn(den, dlu), q));
        ed = __fma_rn(__dmul_rn(s_hdr[d * ns + slot], lm), g2, __dmul_rn(__dmul_rn(den, dld), q));
      }
      sh[r * ns + slot] = w;
      sh[(12 + r) * ns + slot] = eu;
      sh[(24 + r) * ns + slot] = ed;
    }
  }
  // z rows 8 + 2(1 - h) + i from the partner
  double pz[2];
#pragma unroll
  for (int i = 0; i < 2; i++) pz[i] = __shfl_xor_sync(pm, fz[i], 1);
  double *S = a.scratch;
  if (a.needR) {
    // octant o = 4h + ol: x row 2h + (ol >> 1), y row 4 + 2h + (ol & 1),
    // z row 8 + ol; first touch from the x row, then y, then z (row order)
#pragma unroll
    for (int ol = 0; ol < 4; ol++) {
      const double f1 = fx[ol >> 1], f2 = fy[ol & 1];
      const double f3 = ((ol >> 1) == h) ? fz[ol & 1] : pz[ol & 1];
      double Rv = (ol & 1) ? -f1 : f1;
      Rv = (ol & 2) ? Rv - f2 : Rv + f2;
      // (one addition: a predicated one of the other sign takes the pipe as long)
      Rv += __longlong_as_double(__double_as_longlong(f3) ^ ((long long)h << 63));
      S[64 * P + (4 * h + ol) * P + vc] = Rv;
    }
  }
  if (!a.needJ) return;
  // whether any row of this warp's vertices has an E term (the two lanes of a
  // pair have to agree: each reads the E terms of the other's rows)
  const bool with_e = RHO != RHO_CONST || __any_sync(warp, any_e != 0);
  if (RHO == RHO_CONST && with_e) {
#pragma unroll 1
    for (int t = 0; t < 6; t++) {
      const int axis = t >> 1, i = t & 1, r = 4 * axis + 2 * h + i;
      const bool fdn = down >> t & 1;
      const int u = up_octant(axis, i);
      const double dl = s_dlam[(fdn ? u : u + (1 << axis)) * ns + slot];
      const double e = __dmul_rn(__dmul_rn(kRhoConst, sh[(12 + r) * ns + slot]), dl);
      sh[(12 + r) * ns + slot] = fdn ? e : 0.0;
      sh[(24 + r) * ns + slot] = fdn ? 0.0 : e;
    }
  }
  __syncwarp(pm);
#pragma unroll 1
  for (int c = 0; c < 8; c++) {
    // entries jj = 0..3 of this lane are entries j = 4h + jj of octant c
    double wk[3], es[3], en[3], Tk[3][4];
    int bw[3], mb[4];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) mb[jj] = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int r = canon_row(c, k);
      const bool up = canon_is_up(c, k);
      wk[k] = sh[r * ns + slot];
      bw[k] = d_bexp(wk[k]);
      if (with_e) {
        const double eu = sh[(12 + r) * ns + slot], ed = sh[(24 + r) * ns + slot];
        es[k] = up ? eu : ed;  // E term of c itself (entry 0)
        en[k] = up ? ed : eu;  // E term of the neighbour c ^ (1 << k) (entry 1 << k)
      }
      const double *T = a.Tc + (long long)(r * 8) * P + vc;
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        Tk[k][jj] = T[((4 * h + jj) ^ c) * P];
        mb[jj] = max(mb[jj], bw[k] + d_bexp(Tk[k][jj]) - 1023);
      }
      if (!with_e) continue;
      if (k < 2) {
        if (h == 0) {
          mb[0] = max(mb[0], d_bexp(es[k]));
          mb[1 << k] = max(mb[1 << k], d_bexp(en[k]));
        }
      } else {
        mb[0] = max(mb[0], d_bexp(h ? en[2] : es[2]));  // entry 4 gets en[2]
      }
    }
    ff acc[4];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) acc[jj] = ff{0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const bool up = canon_is_up(c, k);
      ff wf = ff_split_scaled(wk[k], bw[k], 1023 - bw[k]);
      if (up) wf = ff_neg(wf);
#pragma unroll
      for (int jj = 0; jj < 4; jj++)
        ff_acc(acc[jj], ff_mul(wf, ff_split_scaled(Tk[k][jj], d_bexp(Tk[k][jj]), bw[k] - mb[jj])));
      if (!with_e) continue;
      const double e0 = h ? en[k] : es[k];
      ff ef = ff_split_scaled(e0, d_bexp(e0), 1023 - mb[0]);
      ff nf = k < 2 ? ff_split_scaled(en[k], d_bexp(en[k]), 1023 - mb[(1 << k) & 3]) : ff{0.0f, 0.0f};
      if (up) {
        ef = ff_neg(ef);
        nf = ff_neg(nf);
      }
      if (h == 0 || k == 2) ff_acc(acc[0], ef);
      if (k < 2 && h == 0) ff_acc(acc[(1 << k) & 3], nf);
    }
    double *dst = S + ((long long)c * P + vc) * 8;
#pragma unroll
    for (int jj = 0; jj < 4; jj++) dst[(4 * h + jj) ^ c] = ff_to_d(acc[jj], mb[jj] - 1023);
  }
}

// ---------------------------------------------------------------------------
// 3. other vertices (boundary, prismatic, irregular): gen_lanes threads each
// (pack_generic).  The
// lanes load the columns' state into shared memory, take the rows (T.P and
// upwinding: FP64, whose instructions cost a warp the same with few lanes
// active as with all), then the entries of J_v.  A cell has three faces at a
// vertex, so an entry has at most three rows; which, with which signs, and the
// cells on their other sides come packed (gen_cell_program).  Every entry
// (c, b) is summed over the rows of cell c in row order, each row's T term
// before its upwind-derivative term.  One warp per vertex with row lists
// built on the fly took 0.41 ms for 108 k prismatic vertices and 0.74 ms for
// 532 k boundary vertices of 512 columns.

// bytes: rows 0-2 (255: none), flags (bit k: the cell is row k's up cell),
// then the local cell on the other side of each row (255: the boundary)
struct GenCell {
  int row[3], other[3];
  unsigned flags;
};
__device__ __forceinline__ GenCell gen_cell(uint2 u) {
  GenCell c;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    c.row[k] = (u.x >> (8 * k)) & 255u;
    c.other[k] = (u.y >> (8 * k)) & 255u;
  }
  c.flags = u.x >> 24;
  return c;
}

template <bool FFJ>
__device__ __forceinline__ void generic_vertex_group(const DevArgs &a, int block) {
  extern __shared__ double sh[];
  const int L = a.gen_lanes, grp = threadIdx.x / L, lane = threadIdx.x & (L - 1);
  const int g = block * (128 / L) + grp;
  if (g >= a.ngen) return;  // whole group
  const unsigned mask = L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
  const GenVertex d = a.gen[g];
  const int *ce = a.g_col + d.col0;
  if (inst_skipped(a, ce[0])) return;  // whole group
  const int nrow = d.nrow, ncol = d.ncol, nint = d.nint, R = a.gen_max_row, C = a.gen_max_col;
  const bool vary = a.rho_type != WATER_DENSITY_CONSTANT;
  const double *T = a.trans + d.trans;
  double *Jv = a.scratch + d.jv;
  // per column: P, kr/mu and its derivative (rho/2 and its derivative where
  // the density varies), seepage; per row: flux, w, E_up, E_dn, exponent of w
  double *sP = sh + (size_t)grp * a.gen_doubles, *sl = sP + C, *sd = sl + C, *sh2 = sd + C, *shd = sh2 + (vary ? C : 0);
  double *fl = shd + (vary ? C : 0), *w = fl + R, *Eu = w + R, *Ed = Eu + R;
  float2 *wf = reinterpret_cast<float2 *>(w);
  int *bw = reinterpret_cast<int *>(Ed + R);
  unsigned char *sp = reinterpret_cast<unsigned char *>(bw + R);
  for (int c = lane; c < ncol; c += L) {
    const int e = ce[c];
    sP[c] = a.P[e];
    sl[c] = a.lam[e];
    sd[c] = a.dlam[e];
    if (vary) {
      sh2[c] = a.hr[e];
      shd[c] = a.hdr[e];
    }
    sp[c] = a.seep[e];
  }
  __syncwarp(mask);
  for (int r = lane; r < nrow; r += L) {
    const double *Tr = T + r * ncol;
    double TP = 0.0;
#pragma unroll 4
    for (int c = 0; c < ncol; c++) TP = __fma_rn(Tr[c], sP[c], TP);
    const uchar2 ud = a.g_rowc[d.row0 + r];
    const int up = ud.x, dn = ud.y;
    const double G = a.g_rowG[d.row0 + r];
    const double den = vary ? __dadd_rn(sh2[up], sh2[dn]) : kRhoConst;
    const double q = __fma_rn(den, G, TP);
    const bool flowdn = dneg(q);
    const int u = flowdn ? up : dn;
    const double lm = sl[u];
    const bool zero = sp[u] != 0;
    const double wr = zero ? 0.0 : vary ? __dmul_rn(den, lm) : lm;
    fl[r] = -__dmul_rn(wr, q);
    if (a.needJ) {
      double eu = 0.0, ed = 0.0;
      if (!zero) {
        if (vary) {
          const double dlu = flowdn ? sd[up] : 0.0, dld = flowdn ? 0.0 : sd[dn];
          const double g2 = q + den * G;
          eu = shd[up] * lm * g2 + den * dlu * q;
          ed = shd[dn] * lm * g2 + den * dld * q;
        } else {
          const double e = __dmul_rn(__dmul_rn(den, sd[u]), q);
          eu = flowdn ? e : 0.0;
          ed = flowdn ? 0.0 : e;
        }
      }
      Eu[r] = eu;
      Ed[r] = ed;
      if (FFJ) {
        const int b = d_bexp(wr);
        const ff f = ff_split_scaled(wr, b, 1023 - b);
        wf[r] = make_float2(f.h, f.l);
        bw[r] = b;
      } else {
        w[r] = wr;
      }
    }
  }
  __syncwarp(mask);
  const uint2 *prog = a.g_cell + d.cell0;
  if (a.needR) {
    for (int c = lane; c < nint; c += L) {
      const GenCell gc = gen_cell(prog[c]);
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (gc.row[k] != 255) s += (gc.flags >> k & 1) ? fl[gc.row[k]] : -fl[gc.row[k]];
      Jv[nint * nint + c] = s;
    }
  }
  if (!a.needJ) return;
  int c = 0, b = lane;
  for (;; b += L) {
    while (b >= nint) {
      b -= nint;
      c++;
    }
    if (c >= nint) break;
    const GenCell gc = gen_cell(prog[c]);
    if (FFJ) {
      // every product at the entry's own power-of-two scale, as for the
      // canonical vertices
      int mb = 0;
      double t[3], e[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        t[k] = e[k] = 0.0;
        if (gc.row[k] == 255) continue;
        const int r = gc.row[k];
        const bool isup = gc.flags >> k & 1;
        t[k] = T[r * ncol + b];
        mb = max(mb, bw[r] + d_bexp(t[k]) - 1023);
        if (b == c || b == gc.other[k]) {
          e[k] = (b == c) == isup ? Eu[r] : Ed[r];
          mb = max(mb, d_bexp(e[k]));
        }
      }
      ff acc = {0.0f, 0.0f};
#pragma unroll
      for (int k = 0; k < 3; k++) {
        if (gc.row[k] == 255) continue;
        const int r = gc.row[k];
        const bool isup = gc.flags >> k & 1;
        const float2 f = wf[r];
        const ff p = ff_mul(ff{f.x, f.y}, ff_split_scaled(t[k], d_bexp(t[k]), bw[r] - mb));
        ff_acc(acc, isup ? ff_neg(p) : p);
        if (b == c || b == gc.other[k]) {
          const ff ef = ff_split_scaled(e[k], d_bexp(e[k]), 1023 - mb);
          ff_acc(acc, isup ? ff_neg(ef) : ef);
        }
      }
      Jv[c * nint + b] = ff_to_d(acc, mb - 1023);
    } else {
      double J = 0.0;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        if (gc.row[k] == 255) continue;
        const int r = gc.row[k];
        const bool isup = gc.flags >> k & 1;
        J = __fma_rn(isup ? -w[r] : w[r], T[r * ncol + b], J);
        if (b == c || b == gc.other[k]) {
          const double et = (b == c) == isup ? Eu[r] : Ed[r];
          J = __dadd_rn(J, isup ? -et : et);
        }
      }
      Jv[c * nint + b] = J;
    }
  }
}

// The other vertices take the first blocks of the canonical vertices' launch,
// so they overlap and the chain of their rows is off the launch's tail.
template <int RHO>
__global__ void __launch_bounds__(128) vertex_kernel(DevArgs a, int gen_blocks) {
  stage_begin();
  if ((int)blockIdx.x >= gen_blocks) {
    const int vc = a.vc0 + ((int)blockIdx.x - gen_blocks) * blockDim.x + threadIdx.x;
    if (vc < a.vc1 && !inst_skipped(a, a.cellc[vc])) canon_vertex_at<RHO>(a, vc, threadIdx.x);
  } else {
    generic_vertex_group<false>(a, blockIdx.x);
  }
}

// The same with a lane pair per canonical vertex (double-float Jacobian
// products): a block of kPairThreads threads takes kPairThreads / 2 vertices.
constexpr int kPairThreads = 128;
template <int RHO>
__global__ void __launch_bounds__(kPairThreads, 7) vertex_pair_kernel(DevArgs a, int gen_blocks) {
  stage_begin();
  if ((int)blockIdx.x >= gen_blocks) {
    const int slot = threadIdx.x >> 1, h = threadIdx.x & 1;
    const int vc = a.vc0 + ((int)blockIdx.x - gen_blocks) * (kPairThreads / 2) + slot;
    const bool on = vc < a.vc1 && !inst_skipped(a, a.cellc[vc]);
    const unsigned warp = RHO == RHO_CONST ? __ballot_sync(0xffffffffu, on) : 0;
    if (on) canon_vertex_pair<RHO>(a, vc, slot, h, kPairThreads / 2, warp);
  } else {
    generic_vertex_group<true>(a, blockIdx.x);
  }
}

template <bool FFJ>
__global__ void __launch_bounds__(128) generic_vertex_kernel(DevArgs a) {
  stage_begin();
  generic_vertex_group<FFJ>(a, blockIdx.x);
}

// ---------------------------------------------------------------------------
// 4. per-cell deterministic gather into R and the CSR row.
//
// Structured interior cells (all vertices canonical, 27-point row) read their
// eight vertices' partials at compile-time slots, one thread each; the others
// follow their gather program.  Both sum the vertices in the cell's corner
// order.

// structured cell sc_cells[sidx]; the 32 lanes of a warp call it together
// with consecutive sidx (those at or past s_end do nothing)
__device__ __forceinline__ void struct_cell_at(const DevArgs &a, int sidx, int s_end) {
  extern __shared__ double rowbuf[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (sidx - lane >= s_end) return;  // whole warp out of range
  bool active = sidx < s_end;
  const int i = active ? a.sc_cells[sidx] : 0;
  active = active && !inst_skipped(a, i);
  if (a.inst_on && !__any_sync(0xffffffffu, active)) return;
  const long long P = a.nCpad, Q = a.nSpad;
  const double *S = a.scratch;
  double row[27];
  if (active) {
    int vc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) vc[j] = a.sc_vc[j * Q + sidx];
    if (a.needR) {
      double s = S[64 * P + d_struct_octant(0) * P + vc[0]];
#pragma unroll
      for (int j = 1; j < 8; j++) s += S[64 * P + d_struct_octant(j) * P + vc[j]];
      s += a.acc_a[i];
      s -= a.acc_b[i];
      a.R[i] = s;
    }
    if (a.needJ) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        // 32-byte loads: with 16-byte ones half of a sector waits in L1 for the
        // next request, and more resident warps made the kernel slower
        const double *blk = S + ((long long)d_struct_octant(j) * P + vc[j]) * 8;
        double v[8];
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(blk));
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[4]), "=d"(v[5]), "=d"(v[6]), "=d"(v[7]) : "l"(blk + 4));
#pragma unroll
        for (int b = 0; b < 8; b++) row[d_struct_slot(j, b)] = first_touch(j, b) ? v[b] : row[d_struct_slot(j, b)] + v[b];
      }
      row[13] += a.jdiag[i];
    }
  }
  if (!a.needJ) return;
  // rows of the warp contiguous in the CSR value array: stage and store
  // coalesced; otherwise every thread stores its own row
  const int rp = active ? a.rowptr[i] : 0;
  const int rp0 = __shfl_sync(0xffffffffu, rp, 0);
  const bool contig = __all_sync(0xffffffffu, active && rp == rp0 + 27 * lane);
  if (contig) {
    // nine slots at a time: shared memory for whole rows (13.8 KB a block)
    // would leave L1 little
    double *buf = rowbuf + warp * 32 * 9;
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int k = 0; k < 9; k++) buf[lane * 9 + k] = row[9 * c + k];
      __syncwarp();
      double *out = a.J + rp0 + 9 * c;
#pragma unroll
      for (int t = 0; t < 9; t++) {
        const int e = lane + 32 * t;
        out[27 * (e / 9) + e % 9] = buf[e];
      }
      __syncwarp();
    }
  } else if (active) {
    double *out = a.J + rp;
#pragma unroll
    for (int k = 0; k < 27; k++) out[k] = row[k];
  }
}

// Other cells: kCellLanes lanes each.  The cell's rows J_v[a] of its vertices
// are copied into shared memory (whole sectors, all in flight together, while
// the entries' words load), then every CSR entry is summed by one lane: its
// contributions come packed in a word or two (MPFAOSetup::ge_code), in the
// cell's corner order, and the entries are sorted by the number of
// contributions, so a pass of the lanes makes few additions (a warp's FP64
// addition costs 57 cycles whatever its active lanes).  The row is stored in
// order.  The residuals, ten additions in a chain, take one lane per cell in
// the block's first warp.  204 k prisms: 0.098 ms (0.174 ms adding vertex
// blocks to the row one by one, a half-warp per cell); 387 k boundary cells of
// 512 columns: 0.13 ms (0.416 ms).
constexpr int kCellLanes = 8;
constexpr int kCellThreads = 128;
constexpr int kCellWords = 8;  // words held per lane: rows of up to 64 entries

__global__ void __launch_bounds__(kCellThreads) generic_cell_kernel(DevArgs a) {
  stage_begin();
  extern __shared__ double rowbuf[];  // per cell: the row, then the vertices' rows
  constexpr int NC = kCellThreads / kCellLanes, L = kCellLanes;
  const int tid = threadIdx.x, grp = tid / L, lane = tid % L, block = blockIdx.x;
  const double *S = a.scratch;
  const int per = a.needJ ? NC : kCellThreads;  // cells of the block
  if (a.needR && tid < per && block * per + tid < a.ngc) {
    const GenCellHead h = a.gc[block * per + tid];
    if (!inst_skipped(a, h.cell)) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = k < h.n ? S[a.gv_r[h.k0 + k]] : 0.0;
      double s = v[0];
#pragma unroll
      for (int k = 1; k < 8; k++)
        if (k < h.n) s += v[k];
      s += a.acc_a[h.cell];
      s -= a.acc_b[h.cell];
      a.R[h.cell] = s;
    }
  }
  if (!a.needJ) return;
  const int g = block * NC + grp;
  GenCellHead h = {0, 0, 0, 0, 0, 0, 0};
  if (g < a.ngc) h = a.gc[g];
  if (g >= a.ngc || inst_skipped(a, h.cell)) h.n = h.rn = 0;  // (the warp stays together)
  long long src = 0;
  unsigned pos = 0;
  if (lane < h.n) {
    src = a.gv_j[h.k0 + lane];
    pos = a.gv_n[h.k0 + lane];
  }
  const bool bytes = a.ge_words == 1;
  unsigned long long w[kCellWords];
  unsigned char slot[kCellWords];
  if (bytes) {
#pragma unroll
    for (int t = 0; t < kCellWords; t++)
      if (lane + L * t < h.rn) {
        w[t] = a.ge_code[h.e0 + lane + L * t];
        slot[t] = a.ge_slot[h.e0 + lane + L * t];
      }
  }
  const double jd = h.rn ? a.jdiag[h.cell] : 0.0;
  const int p0 = h.rn ? a.rowptr[h.cell] : 0;
  double *row = rowbuf + (size_t)grp * (a.max_row_nnz + a.gc_max_vals), *val = row + a.max_row_nnz;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const double *from = S + __shfl_sync(0xffffffffu, src, k, L);
    const unsigned pk = __shfl_sync(0xffffffffu, pos, k, L);
    const unsigned to = (unsigned)__cvta_generic_to_shared(val + (pk & 0xffffu));
    for (int b = lane; b < (int)(pk >> 16); b += L)  // (no columns beyond the last vertex)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 8 * b), "l"(from + b));
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  // (the whole warp together; `on`: the lane has an entry.  An addition whose
  // predicate is off in every lane would still take its 57 cycles: branch)
  auto entry = [&](bool on, unsigned long long w0, unsigned long long w1, int sl) {
    double v[8];
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const unsigned c = bytes ? (unsigned)(w0 >> (8 * k)) & 0xffu : (unsigned)((k < 4 ? w0 : w1) >> (16 * (k % 4))) & 0xffffu;
      v[k] = 0.0;
      if (on && c != (bytes ? 0xffu : 0xffffu)) {
        v[k] = val[c];
        cnt = k + 1;
      }
    }
    double s = v[0];
#pragma unroll
    for (int k = 1; k < 8; k++) {
      if (!__any_sync(0xffffffffu, k < cnt)) break;
      s = k < cnt ? __dadd_rn(s, v[k]) : s;
    }
    if (__any_sync(0xffffffffu, on && sl == h.diag)) s = sl == h.diag ? __dadd_rn(s, jd) : s;
    if (on) row[sl] = s;
  };
  const int most = __reduce_max_sync(0xffffffffu, (int)h.rn);
  if (bytes) {
#pragma unroll
    for (int t = 0; t < kCellWords; t++)
      if (L * t < most) entry(lane + L * t < h.rn, w[t], 0, slot[t]);
  }
  for (int e0 = bytes ? L * kCellWords : 0; e0 < most; e0 += L) {
    const int e = e0 + lane;
    const bool on = e < h.rn;
    const size_t q = (size_t)a.ge_words * (h.e0 + e);
    entry(on, on ? a.ge_code[q] : 0, on && !bytes ? a.ge_code[q + 1] : 0, on ? a.ge_slot[h.e0 + e] : 0);
  }
  __syncwarp();
  double *out = a.J + p0;
  for (int e = lane; e < h.rn; e += L) out[e] = row[e];
}

// At 60 x 220 x 85, this launch and the other cells': 0.208 ms, 4.3 TB/s of
// partials, rows and lists; 0.234 ms with 16-byte loads and whole rows in
// shared memory, 0.22 ms with 80 registers and 24 warps, 0.31 ms with the
// other cells in the same launch (69 registers).
__global__ void __launch_bounds__(64, 8) cell_kernel(DevArgs a) {
  stage_begin();
  struct_cell_at(a, blockIdx.x * blockDim.x + threadIdx.x, a.nS);
}

// ---------------------------------------------------------------------------
// Host side

// Stream-ordered device memory; the pool keeps up to kPoolKeep bytes of
// freed memory for reuse instead of returning it to the driver at every
// synchronisation (a server sets up and destroys handles continuously).
static constexpr unsigned long long kPoolKeep = 8ull << 30;
static constexpr int kMaxDevices = 64;
static std::mutex g_dev_mutex;  // per-device one-time set-up below
static bool g_pool_set[kMaxDevices] = {};

int dmem_alloc(void **p, size_t bytes, void *stream) {
  *p = nullptr;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < kMaxDevices) {
    std::lock_guard<std::mutex> lk(g_dev_mutex);
    if (!g_pool_set[dev]) {
      cudaMemPool_t pool;
      CUDA_TRY(cudaDeviceGetDefaultMemPool(&pool, dev));
      unsigned long long keep = kPoolKeep;
      CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
      g_pool_set[dev] = true;
    }
  }
  cudaError_t e = cudaMallocAsync(p, bytes ? bytes : 1, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    *p = nullptr;
    return set_error(TDY_ERR_GPU, "cudaMallocAsync(%zu bytes): %s", bytes, cudaGetErrorString(e));
  }
  return 0;
}

void dmem_free(void *p, void *stream) {
  if (p) cudaFreeAsync(p, (cudaStream_t)stream);
}

template <class T>
static int dalloc(DeviceState *d, T **p, size_t n) {
  int ierr = dmem_alloc((void **)p, (n ? n : 1) * sizeof(T), d->stream);
  if (ierr) return ierr;
  d->allocs.push_back(*p);
  return 0;
}

static int pool_event(cudaEvent_t *ev);

// Records that a caller's stream enqueued work on this handle.
static int note_stream(DeviceState *d, cudaStream_t st) {
  if (st == d->stream) return 0;
  for (auto &u : d->user_streams)
    if (u.first == st) {
      CUDA_TRY(cudaEventRecord(u.second, st));
      return 0;
    }
  cudaEvent_t e;
  int ierr = pool_event(&e);
  if (ierr) return ierr;
  d->user_streams.emplace_back(st, e);
  CUDA_TRY(cudaEventRecord(e, st));
  return 0;
}

// Slabs of the host-pointer evaluation, for a single extruded block (cells
// numbered layer by layer): cells split at layer boundaries, the first slab
// 1/kSlabFirst of the layers, each next one kSlabGrowth times the previous
// up to 1/kSlabCap (a remainder below half a slab joins the last one).  The
// copies of R and J to host memory run about 1.2x slower than the
// evaluation, so once the first slab is evaluated the copy engine stays
// busy; slabs much thinner than this cost more than they save, since every
// launch lasts at least the latency of one block (about 30 us for the vertex
// stage).  A vertex belongs to the slab of the first cell that uses it, so
// the cells of slab k need only vertices of slabs <= k.  The vertex and cell
// lists (ascending indices) must then run through the slabs in order, which
// is checked: any other numbering leaves one slab (no pipelining).  Slab k
// also computes the state of the cells its vertices read beyond its own (the
// layer above), up to e1.
constexpr double kSlabFirst = 16, kSlabGrowth = 1.25, kSlabCap = 8;
static void build_slabs(_p_TDy *t, DeviceState *d) {
  d->slabs.clear();
  if (t->mesh_blocks.size() != 1) return;
  const ExtrudedInput &blk = t->mesh_blocks[0];
  const Mesh &m = t->mesh;
  const MPFAOSetup &s = t->setup;
  const int nl = blk.nlayers, nc2 = blk.nc2;
  if (nl < 8 || m.nc != nl * nc2) return;
  const double cap = nl / kSlabCap;
  std::vector<int> cut = {0};
  int step = 1;
  for (double size = nl / kSlabFirst, layer = 0; layer < nl; size = std::min(cap, size * kSlabGrowth)) {
    step = std::max(1, (int)std::lround(size));
    layer = std::min<double>(nl, layer + step);
    cut.push_back((int)layer * nc2);
  }
  if (cut.size() > 2 && 2 * (cut[cut.size() - 1] - cut[cut.size() - 2]) < step * nc2) cut.erase(cut.end() - 2);
  const int K = (int)cut.size() - 1;
  if (K < 2) return;
  auto slab_of_cell = [&](int c) { return (int)(std::upper_bound(cut.begin(), cut.end(), c) - cut.begin()) - 1; };
  auto slab_of_vertex = [&](int v) { return slab_of_cell(m.vert_cells[m.vert_cell_off[v]]); };
  // b[k] = first list index in slab k or later; false if the slab decreases
  auto bounds = [&](const std::vector<int> &list, auto slab_of, std::vector<int> &b) {
    b.assign(K + 1, (int)list.size());
    b[0] = 0;
    int cur = 0;
    for (int i = 0; i < (int)list.size(); i++) {
      const int sk = slab_of(list[i]);
      if (sk < cur) return false;
      while (cur < sk) b[++cur] = i;
    }
    return true;
  };
  std::vector<int> bc, bg, bs, bgc;
  if (!bounds(s.canon_vertex, slab_of_vertex, bc) || !bounds(s.gen_vertex, slab_of_vertex, bg) ||
      !bounds(s.sc_cells, slab_of_cell, bs) || !bounds(s.gc_cells, slab_of_cell, bgc))
    return;
  int e_prev = 0;
  for (int k = 0; k < K; k++) {
    DeviceState::Slab sl;
    int need = cut[k + 1];
    auto reach = [&](const std::vector<int> &list, int b0, int b1) {
      for (int i = b0; i < b1; i++) {
        const int v = list[i];
        for (int q = m.vert_cell_off[v]; q < m.vert_cell_off[v + 1]; q++) need = std::max(need, m.vert_cells[q] + 1);
      }
    };
    reach(s.canon_vertex, bc[k], bc[k + 1]);
    reach(s.gen_vertex, bg[k], bg[k + 1]);
    sl.e0 = e_prev;
    sl.e1 = k == K - 1 ? m.nc : std::max(std::min(need, m.nc), e_prev);
    e_prev = sl.e1;
    sl.c0 = cut[k];
    sl.c1 = cut[k + 1];
    sl.vc0 = bc[k];
    sl.vc1 = bc[k + 1];
    sl.g0 = bg[k];
    sl.g1 = bg[k + 1];
    sl.s0 = bs[k];
    sl.s1 = bs[k + 1];
    sl.gc0 = bgc[k];
    sl.gc1 = bgc[k + 1];
    sl.j0 = s.rowptr[cut[k]];
    sl.j1 = s.rowptr[cut[k + 1]];
    d->slabs.push_back(sl);
  }
}

static int noalloc_resolve(int dev);

// Dynamic shared memory above 48 KB is an opt-in per kernel and device; it
// is made at set-up with the device current (and only ever raised).
static size_t g_cell_smem_granted[kMaxDevices] = {};
static size_t gen_cell_smem(const DevArgs &a);
static int cell_smem_optin(int dev, size_t bytes) {
  if (bytes <= 48 * 1024) return 0;
  if (dev < 0 || dev >= kMaxDevices) return set_error(TDY_ERR_SUP, "device ordinal %d not supported", dev);
  std::lock_guard<std::mutex> lk(g_dev_mutex);
  if (bytes > g_cell_smem_granted[dev]) {
    CUDA_TRY(cudaFuncSetAttribute(generic_cell_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    g_cell_smem_granted[dev] = bytes;
  }
  return 0;
}

// Streams and events of handles come from per-device pools and go back to
// them when the handle is destroyed (after their work has completed):
// creating and destroying them waits on the driver, and a server sets up and
// destroys handles on many threads at once.
static std::vector<cudaStream_t> g_stream_pool[kMaxDevices];
static std::vector<cudaEvent_t> g_event_pool[kMaxDevices];

static int pool_device(int *dev) {
  CUDA_TRY(cudaGetDevice(dev));
  if (*dev < 0 || *dev >= kMaxDevices) return set_error(TDY_ERR_SUP, "device ordinal %d not supported", *dev);
  return 0;
}
static int pool_stream(cudaStream_t *st) {
  int dev, ierr;
  if ((ierr = pool_device(&dev))) return ierr;
  {
    std::lock_guard<std::mutex> lk(g_dev_mutex);
    if (!g_stream_pool[dev].empty()) {
      *st = g_stream_pool[dev].back();
      g_stream_pool[dev].pop_back();
      return 0;
    }
  }
  CUDA_TRY(cudaStreamCreateWithFlags(st, cudaStreamNonBlocking));
  return 0;
}
static int pool_event(cudaEvent_t *ev) {
  int dev, ierr;
  if ((ierr = pool_device(&dev))) return ierr;
  {
    std::lock_guard<std::mutex> lk(g_dev_mutex);
    if (!g_event_pool[dev].empty()) {
      *ev = g_event_pool[dev].back();
      g_event_pool[dev].pop_back();
      return 0;
    }
  }
  CUDA_TRY(cudaEventCreateWithFlags(ev, cudaEventDisableTiming));
  return 0;
}
// (dev: the device the stream or event was made on; its work has completed)
static void pool_release(int dev, cudaStream_t st, cudaEvent_t ev) {
  if (dev < 0 || dev >= kMaxDevices) return;
  std::lock_guard<std::mutex> lk(g_dev_mutex);
  if (st) g_stream_pool[dev].push_back(st);
  if (ev) g_event_pool[dev].push_back(ev);
}

int device_pool_stream(cudaStream_t *st) { return pool_stream(st); }
int device_pool_event(cudaEvent_t *ev) { return pool_event(ev); }
void device_pool_release(int dev, cudaStream_t st, cudaEvent_t ev) { pool_release(dev, st, ev); }

// The other vertices' descriptions (GenVertex, gen_cell) in gen_vertex order,
// and the lanes and shared memory they take.
static int pack_generic(const _p_TDy *t, std::vector<GenVertex> &gen, std::vector<int> &g_col,
                        std::vector<double> &g_rowG, std::vector<uchar2> &g_rowc, std::vector<uint2> &g_cell,
                        DevArgs *a) {
  const Mesh &m = t->mesh;
  const MPFAOSetup &s = t->setup;
  int max_row = 1, max_col = 1;
  long long trans = 0;
  gen.reserve(s.gen_vertex.size());
  g_rowG.reserve(s.nrows);
  g_rowc.reserve(s.nrows);
  for (int v : s.gen_vertex) {
    GenVertex d;
    const int r0 = s.v_row_off[v], nrow = s.v_row_off[v + 1] - r0;
    const int c0 = s.v_col_off[v], ncol = s.v_col_off[v + 1] - c0, nint = s.v_nint[v];
    if (ncol > 255) return set_error(TDY_ERR_SUP, "vertex %d has %d columns (max 255)", v, ncol);
    d.trans = s.v_trans_off[v];
    d.jv = s.v_jv_off[v];
    d.row0 = (int)g_rowG.size();
    d.col0 = (int)g_col.size();
    d.cell0 = (int)g_cell.size();
    d.nrow = (unsigned char)nrow;
    d.ncol = (unsigned char)ncol;
    d.nint = (unsigned char)nint;
    d.pad = 0;
    gen.push_back(d);
    g_col.insert(g_col.end(), s.col_ext.begin() + c0, s.col_ext.begin() + c0 + ncol);
    g_cell.insert(g_cell.end(), nint, make_uint2(0x00ffffffu, 0x00ffffffu));
    uint2 *cells = g_cell.data() + d.cell0;
    int count[TDY_MAX_NINT] = {0};
    auto add = [&](int c, int r, bool up, int other) {
      if (c < 0) return true;
      const int k = count[c]++;
      if (k >= 3) return false;
      cells[c].x = (cells[c].x & ~(255u << (8 * k))) | ((unsigned)r << (8 * k)) | (up ? 1u << (24 + k) : 0u);
      cells[c].y = (cells[c].y & ~(255u << (8 * k))) | ((unsigned)(other < 0 ? 255 : other) << (8 * k));
      return true;
    };
    for (int r = 0; r < nrow; r++) {
      const int f = s.row_face[r0 + r], lu = s.row_lup[r0 + r], ld = s.row_ldn[r0 + r];
      // the column of a boundary side: the face's Dirichlet column
      int bc = -1;
      if (lu < 0 || ld < 0)
        for (int c = nint; c < ncol; c++)
          if (s.col_ext[c0 + c] == m.nc + m.face_bnd[f]) bc = c;
      if ((lu < 0 || ld < 0) && bc < 0) return set_error(TDY_ERR_LIB, "vertex %d: row without its boundary column", v);
      g_rowG.push_back(s.gravdis[f]);
      g_rowc.push_back(make_uchar2((unsigned char)(lu < 0 ? bc : lu), (unsigned char)(ld < 0 ? bc : ld)));
      if (!add(lu, r, true, ld) || !add(ld, r, false, lu))
        return set_error(TDY_ERR_SUP, "vertex %d: a cell with more than 3 rows", v);
    }
    max_row = std::max(max_row, nrow);
    max_col = std::max(max_col, ncol);
    trans += (long long)nrow * ncol;
  }
  a->ngen = (int)gen.size();
  a->gen_max_row = max_row;
  a->gen_max_col = max_col;
  // per column 3 doubles (5 where the density varies) and a byte; per row 4
  // doubles and an int
  const bool vary = a->rho_type != WATER_DENSITY_CONSTANT;
  a->gen_doubles = (vary ? 5 : 3) * max_col + 4 * max_row + (4 * max_row + max_col + 7) / 8;
  // 4 lanes where a vertex's Trans is small (hexahedra's boundary: 13 to 27
  // elements), a warp where it is large (prisms: 107 to 205): it is read for
  // the rows and again for J_v, and more vertices in flight push it out of L1.
  // F and J in us with 4, 8, 32 lanes: 8 columns 39, 40, 52; 128 columns 173,
  // 194, 306; 512 columns 582, 653, 1125; 60 x 110 x 40 cells 224, 229, 258; 31 x
  // 57 x 23 cells 66, 62, 73; 500 prisms 61, 61, 29; 20 k 127, 127, 69; 204 k
  // 612, 611, 518.  Nothing measured lies between 27 and 107.
  // A launch of their own where they are many and the most (fewer registers),
  // not where a launch costs more.  F and J in us in the canonical launch and
  // in one of their own, with the lanes above: 8 columns (6.1 k other
  // vertices) 39, 47; 32 columns (30 k) 63, 62; 128 columns (128 k) 173, 179;
  // 512 columns (532 k) 582, 557; prisms with 12 k 69, 66; 23 k 126, 124; 108 k
  // 518, 436; 60 x 110 x 40 cells (27 k, and 251 k canonical ones) 224, 236.
  a->gen_lanes = trans <= 64LL * a->ngen ? 4 : 32;
  a->gen_apart = a->ngen > s.nC && a->ngen > 20000;
  while (a->gen_lanes < 32 && (size_t)(128 / a->gen_lanes) * a->gen_doubles * sizeof(double) > 40 * 1024) a->gen_lanes *= 2;
  return 0;
}

int device_setup(_p_TDy *t) {
  const Mesh &m = t->mesh;
  const MPFAOSetup &s = t->setup;
  if (s.max_nrow > TDY_MAX_ROWS || s.max_nint > TDY_MAX_NINT || s.max_row_nnz > TDY_MAX_ROW_NNZ)
    return set_error(TDY_ERR_SUP,
                     "mesh exceeds kernel limits (rows/vertex %d, cells/vertex %d, row nnz %d; max %d, %d, %d)",
                     s.max_nrow, s.max_nint, s.max_row_nnz, TDY_MAX_ROWS, TDY_MAX_NINT, TDY_MAX_ROW_NNZ);
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return set_error(TDY_ERR_GPU, "no CUDA device available: %s", e != cudaSuccess ? cudaGetErrorString(e) : "0 devices");
  DeviceState *d = new DeviceState();
  t->dev = d;
  CUDA_TRY(cudaGetDevice(&d->device));
  int ierr = 0;
  if ((ierr = pool_stream(&d->stream))) return ierr;
  DevArgs &a = d->a;
  memset(&a, 0, sizeof(a));
  a.nc = m.nc;
  a.nb = m.nb;
  a.nv = m.nv;
  a.Pref = t->opt.Pref;
  a.rho_type = t->opt.rho_type;
  a.mu_type = t->opt.mu_type;
  const int next = m.nc + m.nb;
  // every array of the handle in one allocation, uploaded with one copy
  Arena ar;
  ar.up(&a.vol, m.cell_vol);
  ar.up(&a.poro, t->mat.porosity);
  ar.up(&a.Sr, t->mat.Sr);
  // (van Genuchten: the third slot holds n = 1 / (1 - m))
  std::vector<double> sat_param = t->mat.sat_param;
  for (int c = 0; c < m.nc; c++)
    if (t->mat.sat_type[c] == SAT_FUNC_VAN_GENUCHTEN) sat_param[3 * (size_t)c + 2] = 1.0 / (1.0 - sat_param[3 * (size_t)c]);
  ar.up(&a.sat_param, sat_param);
  ar.up(&a.rp_param, t->mat.relperm_param);
  ar.up(&a.ss, t->mat.source_sink);
  ar.up(&a.sat_type, t->mat.sat_type);
  ar.up(&a.rp_type, t->mat.relperm_type);
  ar.up(&a.lam_sat, t->mat.lam_sat);
  a.vis = t->mat.vis;
  a.inv_vis = 1.0 / t->mat.vis;
  std::vector<int> bnd_cell(m.nb);
  for (int b = 0; b < m.nb; b++) bnd_cell[b] = m.face_cell1[m.bnd_face[b]];
  ar.up(&a.bnd_cell, bnd_cell);
  ar.up(&a.bnd_type, t->bnd.type);
  ar.up(&a.bnd_has, t->bnd.has_value);
  ar.up(&a.bnd_val, t->bnd.value);
  ar.up(&a.bnd_rho, t->bnd.rho);
  ar.up(&a.bnd_vis, t->bnd.vis);
  ar.up(&a.G, s.gravdis);
  a.nC = s.nC;
  a.vc0 = 0;
  a.vc1 = s.nC;
  a.nCpad = s.nCpad;
  if (t->opt.setup_on_device)
    ar.work(&a.Tc, 96 * (size_t)s.nCpad);
  else
    ar.up(&a.Tc, s.Tc);
  a.jac_ff = t->opt.jacobian_arithmetic == JACOBIAN_DOUBLE_FLOAT;
  ar.up(&a.cellc, s.cellc);
  ar.up(&a.facec, s.facec);
  std::vector<GenVertex> gen;
  std::vector<int> g_col;
  std::vector<double> g_rowG;
  std::vector<uchar2> g_rowc;
  std::vector<uint2> g_cell;
  if ((ierr = pack_generic(t, gen, g_col, g_rowG, g_rowc, g_cell, &a))) return ierr;
  ar.up(&a.gen, gen);
  ar.up(&a.g_col, g_col);
  ar.up(&a.g_rowG, g_rowG);
  ar.up(&a.g_rowc, g_rowc);
  ar.up(&a.g_cell, g_cell);
  ar.up(&a.trans, s.trans);
  ar.up(&a.rowptr, s.rowptr);
  std::vector<GenCellHead> gc(s.gc_cells.size());
  for (size_t g = 0; g < gc.size(); g++) {
    const int c = s.gc_cells[g];
    gc[g] = GenCellHead{c, s.gv_off[g], s.ge_off[g], (unsigned char)(s.gv_off[g + 1] - s.gv_off[g]),
                        (unsigned char)(s.rowptr[c + 1] - s.rowptr[c]), s.gc_diag[g], 0};
  }
  ar.up(&a.gc, gc);
  ar.up(&a.gv_j, s.gv_j);
  ar.up(&a.gv_r, s.gv_r);
  ar.up(&a.gv_n, s.gv_n);
  ar.up(&a.ge_code, s.ge_code);
  ar.up(&a.ge_slot, s.ge_slot);
  a.ge_words = s.ge_words;
  a.gc_max_vals = s.gc_max_vals;
  a.max_row_nnz = s.max_row_nnz;
  a.nS = s.nS;
  a.nSpad = s.nSpad;
  a.ngc = (int)s.gc_cells.size();
  ar.up(&a.sc_cells, s.sc_cells);
  ar.up(&a.sc_vc, s.sc_vc);
  ar.work(&a.P, next);
  ar.work(&a.hr, a.rho_type == WATER_DENSITY_CONSTANT ? 0 : next);
  ar.work(&a.hdr, a.rho_type == WATER_DENSITY_CONSTANT ? 0 : next);
  ar.work(&a.lam, next);
  ar.work(&a.dlam, next);
  ar.work(&a.seep, next);
  ar.work(&a.acc_a, m.nc);
  ar.work(&a.acc_b, m.nc);
  ar.work(&a.jdiag, m.nc);
  double *accum_prev = nullptr;
  ar.work(&accum_prev, m.nc);
  ar.work(&a.scratch, (size_t)s.scratch_size);
  d->nnz = (int)s.colidx.size();
  ar.work(&d->dU, m.nc);
  ar.work(&d->dUt, m.nc);
  ar.work(&d->dR, m.nc);
  ar.work(&d->dJ, d->nnz);
  ar.work(&d->diagS, m.nc);
  ar.work(&d->diagMass, m.nc);
  d->inst_ok = s.max_row_nnz <= 96;  // (the interface's limit; the stages themselves have none)
  std::vector<int> cell_inst;
  if (t->mesh_blocks.size() > 1) {
    for (size_t b = 0; b < t->mesh_blocks.size(); b++)
      cell_inst.insert(cell_inst.end(), (size_t)t->mesh_blocks[b].nc2 * t->mesh_blocks[b].nlayers, (int)b);
    ar.up(&a.cell_inst, cell_inst);
    ar.work(&d->inst_on, t->mesh_blocks.size());
  }
  if ((ierr = ar.commit(d->stream))) return ierr;
  d->allocs.push_back(ar.base);
  CUDA_TRY(cudaMemsetAsync(accum_prev, 0, sizeof(double) * m.nc, d->stream));
  // what no evaluation changes: no cell seeps
  CUDA_TRY(cudaMemsetAsync(a.seep, 0, next, d->stream));
  a.accum_prev = accum_prev;
  if (t->opt.setup_on_device &&
      (ierr = device_canon_trans(t, a.cellc, a.facec, const_cast<double *>(a.Tc), d->stream)))
    return ierr;
  if (t->opt.setup_on_device && (ierr = device_gen_trans(t, const_cast<double *>(a.trans), d->stream))) return ierr;
  build_slabs(t, d);  // their copy stream and events are taken on first use
  if ((ierr = cell_smem_optin(d->device, gen_cell_smem(a)))) return ierr;
  if ((ierr = noalloc_resolve(d->device))) return ierr;
  if ((ierr = pool_event(&d->noalloc_ev))) return ierr;
  // the uploads (and the device-built Trans) are complete before any other
  // stream uses them, and the staging buffer and host vectors above outlive
  // them; only this handle's stream is waited for
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

// Waits for the work this handle has in flight (its own streams and the
// callers' streams it has seen), frees its memory stream-ordered (no
// device-wide synchronisation, so other handles keep running) and returns its
// streams and events to the pools.
void device_destroy(_p_TDy *t) {
  DeviceState *d = t->dev;
  if (!d) return;
  if (d->stream) cudaStreamSynchronize(d->stream);
  for (auto &u : d->user_streams) {
    cudaEventSynchronize(u.second);
    pool_release(d->device, nullptr, u.second);
  }
  if (d->noalloc_ev) {
    cudaEventSynchronize(d->noalloc_ev);
    pool_release(d->device, nullptr, d->noalloc_ev);
  }
  for (int k = 0; k < 4; k++)
    if (d->ev[k]) cudaEventDestroy(d->ev[k]);
  if (d->slab_exec) cudaGraphExecDestroy(d->slab_exec);
  if (d->copy_stream) {
    cudaStreamSynchronize(d->copy_stream);
    pool_release(d->device, d->copy_stream, nullptr);
  }
  for (cudaEvent_t e : d->slab_ev) pool_release(d->device, nullptr, e);
  if (d->stream) {
    for (void *p : d->allocs) dmem_free(p, d->stream);
    cudaStreamSynchronize(d->stream);
    pool_release(d->device, d->stream, nullptr);
  }
  delete d;
  t->dev = nullptr;
}

int device_upload_source_sink(_p_TDy *t) {
  DeviceState *d = t->dev;
  CUDA_TRY(cudaMemcpyAsync((void *)d->a.ss, t->mat.source_sink.data(), sizeof(double) * t->mesh.nc,
                           cudaMemcpyHostToDevice, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

static inline unsigned nblocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// A multiplier coprime to n near 0.618 n (golden-ratio stride), so that
// chunk -> chunk * m mod n is a permutation that scatters neighbouring chunks.
static int chunk_multiplier(int n) {
  if (n <= 2) return 1;
  long long m = (long long)(0.6180339887 * n) | 1;
  auto gcd = [](long long x, long long y) {
    while (y) {
      long long t = x % y;
      x = y;
      y = t;
    }
    return x;
  };
  while (gcd(m, n) != 1) m += 2;
  return (int)(m % n);
}

int device_presolve(_p_TDy *t, const double *dUprev, void *stream, bool fp64_curves) {
  DeviceState *d = t->dev;
  cudaStream_t st = stream ? (cudaStream_t)stream : d->stream;
  DevArgs a = d->a;
  a.dt = t->dtime;
  a.fp64_curves = fp64_curves;
  presolve_kernel<<<nblocks(a.nc, 256), 256, 0, st>>>(a, dUprev, (double *)a.accum_prev);
  CUDA_TRY(cudaGetLastError());
  return note_stream(d, st);
}

int device_presolve_host(_p_TDy *t, const double *Uprev) {
  DeviceState *d = t->dev;
  CUDA_TRY(cudaMemcpyAsync(d->dU, Uprev, sizeof(double) * t->mesh.nc, cudaMemcpyHostToDevice, d->stream));
  int ierr = device_presolve(t, d->dU, d->stream);
  if (ierr) return ierr;
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

static void launch_state_range(const DevArgs &a, int e0, int e1, Emit &e) {
  if (e1 <= e0) return;
  const int nchunks = (int)nblocks(e1 - e0, 32);
  e(state_kernel, nblocks((long long)nchunks * 32, 256), 256, 0, a, e0, e1, nchunks, chunk_multiplier(nchunks));
}
static void launch_state(const DevArgs &a, Emit &e) { launch_state_range(a, 0, a.nc + a.nb, e); }

// Vertex stage over the vertices a names (gen/ngen, [vc0, vc1)).
static int rho_mode(const DevArgs &a) {
  return a.rho_type == WATER_DENSITY_CONSTANT ? RHO_CONST
         : a.rho_type == WATER_DENSITY_EXPONENTIAL ? RHO_EXP
                                                   : RHO_NODERIV;
}

static void launch_vertices(const DevArgs &a, Emit &e) {
  const int rho = rho_mode(a), per = 128 / a.gen_lanes;
  int gb = (int)nblocks(a.ngen, per);
  size_t gen_smem = gb ? (size_t)per * a.gen_doubles * sizeof(double) : 0;
  if (a.gen_apart) {
    e(a.jac_ff ? generic_vertex_kernel<true> : generic_vertex_kernel<false>, gb, 128, gen_smem, a);
    gb = 0;
    gen_smem = 0;
  }
  if (a.jac_ff) {
    static_assert(kPairThreads == 128, "blocks of the other vertices");
    const int pb = (int)nblocks(a.vc1 - a.vc0, kPairThreads / 2);
    const size_t smem = pb ? (size_t)pair_shared_rows(rho) * (kPairThreads / 2) * sizeof(double) : 0;
    auto k = rho == RHO_CONST ? vertex_pair_kernel<RHO_CONST>
             : rho == RHO_NODERIV ? vertex_pair_kernel<RHO_NODERIV>
                                  : vertex_pair_kernel<RHO_EXP>;
    e(k, pb + gb, kPairThreads, std::max(smem, gen_smem), a, gb);
    return;
  }
  const int cb = (int)nblocks(a.vc1 - a.vc0, 128);
  const size_t smem = cb ? 36 * 128 * sizeof(double) : 0;
  auto k = rho == RHO_CONST ? vertex_kernel<RHO_CONST>
           : rho == RHO_NODERIV ? vertex_kernel<RHO_NODERIV>
                                : vertex_kernel<RHO_EXP>;
  e(k, cb + gb, 128, std::max(smem, gen_smem), a, gb);
}

// Cell stage over the cells a names (sc_cells/nS, gc/ngc).
static size_t gen_cell_smem(const DevArgs &a) {
  return (size_t)(kCellThreads / kCellLanes) * (a.max_row_nnz + a.gc_max_vals) * sizeof(double);
}

static void launch_cells(const DevArgs &a, Emit &e) {
  e(cell_kernel, nblocks(a.nS, 64), 64, 64 * 9 * sizeof(double), a);
  e(generic_cell_kernel, nblocks(a.ngc, a.needJ ? kCellThreads / kCellLanes : kCellThreads), kCellThreads,
    a.needJ ? gen_cell_smem(a) : 0, a);
}

// The stages of one evaluation; events[] (4 entries, or null) bracket them
// for the per-kernel timers.
static int launch_eval(const DevArgs &a, cudaStream_t st, cudaEvent_t *events) {
  Emit e(st);
  if (events) CUDA_TRY(cudaEventRecord(events[0], st));
  launch_state(a, e);
  e.overlap = true;  // (behind an event record the stages follow as before)
  if (events) CUDA_TRY(cudaEventRecord(events[1], st));
  launch_vertices(a, e);
  if (events) CUDA_TRY(cudaEventRecord(events[2], st));
  launch_cells(a, e);
  if (events) CUDA_TRY(cudaEventRecord(events[3], st));
  CUDA_TRY(cudaGetLastError());
  return 0;
}

// The arguments of one evaluation.
static int eval_args(_p_TDy *t, int form, const double *dU, const double *dUt, double shift, double *dR, double *dJ,
                     DevArgs *out, bool fp64_curves = false) {
  DeviceState *d = t->dev;
  if (form == FORM_SNES && !(t->dtime > 0.0))
    return set_error(TDY_ERR_USER, "SNES form needs TDySetDtimeForSNESSolver before evaluation");
  DevArgs a = d->a;
  a.form = form;
  a.U = dU;
  a.Ut = dUt;
  a.dt = t->dtime;
  a.shift = form == FORM_SNES ? 1.0 / t->dtime : shift;
  a.needR = dR != nullptr;
  a.needJ = dJ != nullptr;
  a.R = dR;
  a.J = dJ;
  a.fp64_curves = fp64_curves;
  *out = a;
  return 0;
}

int device_eval(_p_TDy *t, int form, double time, const double *dU, const double *dUt, double shift, double *dR,
                double *dJ, void *stream, bool fp64_curves) {
  (void)time;
  DeviceState *d = t->dev;
  cudaStream_t st = stream ? (cudaStream_t)stream : d->stream;
  DevArgs a;
  int ierr = eval_args(t, form, dU, dUt, shift, dR, dJ, &a, fp64_curves);
  if (ierr) return ierr;
  ierr = launch_eval(a, st, d->timers ? d->ev : nullptr);
  if (ierr) return ierr;
  if ((ierr = note_stream(d, st))) return ierr;
  if (d->timers) {
    CUDA_TRY(cudaEventSynchronize(d->ev[3]));
    for (int k = 0; k < 3; k++) {
      float ms = 0.f;
      CUDA_TRY(cudaEventElapsedTime(&ms, d->ev[k], d->ev[k + 1]));
      d->t_ms[k] += ms;
      d->t_calls[k] += 1;
    }
  }
  return 0;
}

// Evaluation (SNES form) of the listed instances (blocks): the three stages
// with the other instances' entities skipped, which keep their R and J.  The
// skipped threads cost a load and a test each; one CTA per instance, which no
// launch outlasts, took longer than an evaluation of every instance.
int device_eval_instances(_p_TDy *t, const double *dU, double *dR, double *dJ, const int *list, int nlist,
                          void *stream, bool fp64_curves) {
  DeviceState *d = t->dev;
  if (!d->inst_ok) return set_error(TDY_ERR_SUP, "rows of more than 96 entries: no evaluation of single instances");
  if (nlist <= 0) return 0;
  cudaStream_t st = stream ? (cudaStream_t)stream : d->stream;
  DevArgs a;
  int ierr = eval_args(t, FORM_SNES, dU, nullptr, 0.0, dR, dJ, &a, fp64_curves);
  if (ierr) return ierr;
  if (d->inst_on) {
    d->h_on.assign(t->mesh_blocks.size(), 0);
    for (int k = 0; k < nlist; k++) d->h_on[list[k]] = 1;
    CUDA_TRY(cudaMemcpyAsync(d->inst_on, d->h_on.data(), sizeof(int) * d->h_on.size(), cudaMemcpyHostToDevice, st));
    a.inst_on = d->inst_on;
  }
  if ((ierr = launch_eval(a, st, nullptr))) return ierr;
  return note_stream(d, st);
}

bool device_inst_ok(_p_TDy *t) { return t->dev && t->dev->inst_ok; }

void *device_default_stream(_p_TDy *t) { return t->dev ? (void *)t->dev->stream : nullptr; }

int device_download_trans(_p_TDy *t, std::vector<double> &trans) {
  const DeviceState *d = t->dev;
  trans.resize(t->setup.trans.size());
  if (!trans.empty())
    CUDA_TRY(cudaMemcpy(trans.data(), d->a.trans, sizeof(double) * trans.size(), cudaMemcpyDeviceToHost));
  return 0;
}

int device_download_tc(_p_TDy *t, std::vector<double> &Tc) {
  const DeviceState *d = t->dev;
  Tc.resize(96 * (size_t)t->setup.nCpad);
  CUDA_TRY(cudaMemcpy(Tc.data(), d->a.Tc, sizeof(double) * Tc.size(), cudaMemcpyDeviceToHost));
  return 0;
}

int device_set_timers(_p_TDy *t, int on) {
  DeviceState *d = t->dev;
  if (on && !d->ev[0])
    for (int k = 0; k < 4; k++) CUDA_TRY(cudaEventCreate(&d->ev[k]));
  d->timers = on != 0;
  for (int k = 0; k < 3; k++) {
    d->t_ms[k] = 0.0;
    d->t_calls[k] = 0;
  }
  return 0;
}

int device_get_timers(_p_TDy *t, int *n, const char **names, double *ms, long long *calls) {
  DeviceState *d = t->dev;
  int cap = *n;
  *n = 3;
  for (int k = 0; k < 3 && k < cap; k++) {
    if (names) names[k] = kKernelNames[k];
    if (ms) ms[k] = d->t_ms[k];
    if (calls) calls[k] = d->t_calls[k];
  }
  return 0;
}

// FP64 throughput probe: independent FMA chains per thread, enough blocks to
// fill every SM; reports achieved double-precision TFLOP/s on the device.
__global__ void __launch_bounds__(256) fp64_probe_kernel(double *out, int iters) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-9, a2 = a0 + 2e-9, a3 = a0 + 3e-9;
  double a4 = a0 + 4e-9, a5 = a0 + 5e-9, a6 = a0 + 6e-9, a7 = a0 + 7e-9;
  const double b = 0.999999999, c = 1e-12;
  for (int i = 0; i < iters; i++) {
    a0 = fma(a0, b, c);
    a1 = fma(a1, b, c);
    a2 = fma(a2, b, c);
    a3 = fma(a3, b, c);
    a4 = fma(a4, b, c);
    a5 = fma(a5, b, c);
    a6 = fma(a6, b, c);
    a7 = fma(a7, b, c);
  }
  double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.678) out[blockIdx.x] = s;  // keep the chains live
}

int device_fp64_probe(double *tflops) {
  int dev = 0, nsm = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  double *out = nullptr;
  CUDA_TRY(cudaMalloc(&out, sizeof(double) * nsm * 8));
  cudaEvent_t e0, e1;
  CUDA_TRY(cudaEventCreate(&e0));
  CUDA_TRY(cudaEventCreate(&e1));
  const int iters = 4096, blocks = nsm * 8, threads = 256;
  fp64_probe_kernel<<<blocks, threads>>>(out, iters);  // warm-up
  CUDA_TRY(cudaEventRecord(e0));
  const int reps = 5;
  for (int r = 0; r < reps; r++) fp64_probe_kernel<<<blocks, threads>>>(out, iters);
  CUDA_TRY(cudaEventRecord(e1));
  CUDA_TRY(cudaEventSynchronize(e1));
  float ms = 0.f;
  CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  double flops = 2.0 * 8.0 * iters * (double)blocks * threads * reps;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return 0;
}

int device_transient_variable_host(_p_TDy *t, const double *U, double *C, double *dC) {
  DeviceState *d = t->dev;
  const size_t n = (size_t)t->mesh.nc;
  CUDA_TRY(cudaMemcpyAsync(d->dU, U, sizeof(double) * n, cudaMemcpyHostToDevice, d->stream));
  tv_kernel<<<nblocks(n, 256), 256, 0, d->stream>>>(d->a, d->dU, C ? d->diagS : nullptr, dC ? d->diagMass : nullptr);
  CUDA_TRY(cudaGetLastError());
  if (C) CUDA_TRY(cudaMemcpyAsync(C, d->diagS, sizeof(double) * n, cudaMemcpyDeviceToHost, d->stream));
  if (dC) CUDA_TRY(cudaMemcpyAsync(dC, d->diagMass, sizeof(double) * n, cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

int device_eval_dae_host(_p_TDy *t, double time, const double *U2, const double *Ut2, double *R2) {
  DeviceState *d = t->dev;
  const int n = t->mesh.nc;
  if (!d->dae) {  // interleaved buffers, allocated on the first DAE call
    int ierr;
    if ((ierr = dalloc(d, &d->dae, 6 * (size_t)n))) return ierr;
  }
  double *dU2 = d->dae, *dUt2 = d->dae + 2 * (size_t)n, *dR2 = d->dae + 4 * (size_t)n;
  CUDA_TRY(cudaMemcpyAsync(dU2, U2, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, d->stream));
  CUDA_TRY(cudaMemcpyAsync(dUt2, Ut2, sizeof(double) * 2 * n, cudaMemcpyHostToDevice, d->stream));
  dae_split_kernel<<<nblocks(n, 256), 256, 0, d->stream>>>(n, dU2, dUt2, d->dU, d->dUt);
  CUDA_TRY(cudaGetLastError());
  int ierr = device_eval(t, FORM_TV, time, d->dU, d->dUt, 0.0, d->dR, nullptr, d->stream);
  if (ierr) return ierr;
  tv_kernel<<<nblocks(n, 256), 256, 0, d->stream>>>(d->a, d->dU, d->diagS, nullptr);
  dae_merge_kernel<<<nblocks(n, 256), 256, 0, d->stream>>>(n, dU2, d->dR, d->diagS, dR2);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaMemcpyAsync(R2, dR2, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

// The arguments of slab k: the vertices and cells of slab k only.
static DevArgs slab_args(const DevArgs &a, const DeviceState::Slab &sl) {
  DevArgs b = a;
  b.gen = a.gen + sl.g0;
  b.ngen = sl.g1 - sl.g0;
  b.vc0 = sl.vc0;
  b.vc1 = sl.vc1;
  b.sc_cells = a.sc_cells + sl.s0;
  b.sc_vc = a.sc_vc + sl.s0;  // structure of arrays, stride nSpad: the offset carries over
  b.nS = sl.s1 - sl.s0;
  b.gc = a.gc + sl.gc0;
  b.ngc = sl.gc1 - sl.gc0;
  return b;
}

static bool pinned(const void *p) {
  if (!p) return true;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeHost;
}

// The slab pipeline as a graph: U (and U_t) to the device, the boundary
// faces' state, then per slab the state of the cells its vertices read, its
// vertex and cell stages, and its rows of J and R to host memory.  The state
// of slab k waits for that of slab k-1 and, so that the first slab runs
// alone, for the vertex stage of slab k-1; the vertex stage of slab k waits
// for the state of slab k (so it sees every cell it reads); the cell stage of slab k waits
// for its vertex stage only, so it runs beside the state and vertex stages of
// slab k+1 (each stage writes entries no other running stage reads) and the
// tail of one launch overlaps the next; the copies form a chain of their
// own, each after its slab's cell stage, and run while the next slabs are
// evaluated.  One launch replaces about ten driver calls per slab.
static int build_slab_graph(_p_TDy *t, DeviceState *d, const DevArgs &a, const double *U, const double *Ut,
                            double *R, double *J, cudaGraphExec_t *out) {
  const size_t n = (size_t)t->mesh.nc;
  cudaGraph_t g = nullptr;
  CUDA_TRY(cudaGraphCreate(&g, 0));
  cudaError_t err = cudaSuccess;
  cudaGraphNode_t up[2] = {nullptr, nullptr}, join = nullptr, copy_last = nullptr;
  int nup = 0;
  err = cudaGraphAddMemcpyNode1D(&up[nup++], g, nullptr, 0, d->dU, U, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (err == cudaSuccess && Ut)
    err = cudaGraphAddMemcpyNode1D(&up[nup++], g, nullptr, 0, d->dUt, Ut, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (err == cudaSuccess) err = cudaGraphAddEmptyNode(&join, g, up, nup);
  Emit e(nullptr);
  e.g = g;
  e.last = join;
  if (err == cudaSuccess) {
    const size_t K = d->slabs.size();
    launch_state_range(a, a.nc, a.nc + a.nb, e);  // boundary faces
    cudaGraphNode_t sprev = e.last, vprev = nullptr;
    for (size_t k = 0; k < K && err == cudaSuccess && e.err == cudaSuccess; k++) {
      const DeviceState::Slab &sl = d->slabs[k];
      const DevArgs b = slab_args(a, sl);
      // the state of slab k after that of slab k-1 and the vertex stage of
      // slab k-1 (so the first slab runs alone), then its vertex stage
      cudaGraphNode_t sdeps[2] = {sprev, vprev}, sjoin = nullptr;
      err = cudaGraphAddEmptyNode(&sjoin, g, sdeps, vprev ? 2 : 1);
      if (err != cudaSuccess) break;
      e.last = sjoin;
      launch_state_range(a, sl.e0, sl.e1, e);
      sprev = e.last;
      launch_vertices(b, e);
      vprev = e.last;
      launch_cells(b, e);
      if (e.err != cudaSuccess) break;
      cudaGraphNode_t deps[2] = {e.last, copy_last}, nj = nullptr;
      err = cudaGraphAddMemcpyNode1D(&nj, g, deps, copy_last ? 2 : 1, J + sl.j0, d->dJ + sl.j0,
                                     sizeof(double) * (size_t)(sl.j1 - sl.j0), cudaMemcpyDeviceToHost);
      copy_last = nj;
      if (err == cudaSuccess && R) {
        cudaGraphNode_t dr[2] = {e.last, copy_last}, nr = nullptr;
        err = cudaGraphAddMemcpyNode1D(&nr, g, dr, 2, R + sl.c0, d->dR + sl.c0, sizeof(double) * (size_t)(sl.c1 - sl.c0),
                                       cudaMemcpyDeviceToHost);
        copy_last = nr;
      }
    }
  }
  if (err == cudaSuccess) err = e.err;
  if (err == cudaSuccess) err = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (err != cudaSuccess) return set_error(TDY_ERR_GPU, "slab graph: %s", cudaGetErrorString(err));
  return 0;
}

int device_eval_host(_p_TDy *t, int form, double time, const double *U, const double *Ut, double shift, double *R,
                     double *J) {
  DeviceState *d = t->dev;
  const size_t n = (size_t)t->mesh.nc;
  if (d->slabs.size() > 1 && J && !d->timers) {
    // slab by slab (build_slabs): the same launches, split; the same bits
    DevArgs a;
    int ierr = eval_args(t, form, d->dU, Ut ? d->dUt : nullptr, shift, R ? d->dR : nullptr, d->dJ, &a);
    if (ierr) return ierr;
    DeviceState::SlabKey key;
    key.form = form;
    key.dt = a.dt;
    key.shift = a.shift;
    key.U = U;
    key.Ut = Ut;
    key.R = R;
    key.J = J;
    if (d->slab_exec && !(key == d->slab_key)) {
      CUDA_TRY(cudaGraphExecDestroy(d->slab_exec));
      d->slab_exec = nullptr;
    }
    if (!d->slab_exec && pinned(U) && pinned(Ut) && pinned(R) && pinned(J)) {
      if ((ierr = build_slab_graph(t, d, a, U, Ut, R, J, &d->slab_exec))) return ierr;
      d->slab_key = key;
    }
    if (d->slab_exec) {
      CUDA_TRY(cudaGraphLaunch(d->slab_exec, d->stream));
      CUDA_TRY(cudaStreamSynchronize(d->stream));
      return 0;
    }
    // pageable host buffers: the same pipeline on two streams
    CUDA_TRY(cudaMemcpyAsync(d->dU, U, sizeof(double) * n, cudaMemcpyHostToDevice, d->stream));
    if (Ut) CUDA_TRY(cudaMemcpyAsync(d->dUt, Ut, sizeof(double) * n, cudaMemcpyHostToDevice, d->stream));
    if (!d->copy_stream) {  // first such call of this handle
      if ((ierr = pool_stream(&d->copy_stream))) return ierr;
      d->slab_ev.assign(d->slabs.size(), nullptr);
      for (cudaEvent_t &e : d->slab_ev)
        if ((ierr = pool_event(&e))) return ierr;
    }
    Emit e(d->stream);
    launch_state_range(a, a.nc, a.nc + a.nb, e);  // boundary faces
    for (size_t k = 0; k < d->slabs.size(); k++) {
      const DeviceState::Slab &sl = d->slabs[k];
      const DevArgs b = slab_args(a, sl);
      launch_state_range(a, sl.e0, sl.e1, e);
      launch_vertices(b, e);
      launch_cells(b, e);
      CUDA_TRY(cudaEventRecord(d->slab_ev[k], d->stream));
      CUDA_TRY(cudaStreamWaitEvent(d->copy_stream, d->slab_ev[k], 0));
      CUDA_TRY(cudaMemcpyAsync(J + sl.j0, d->dJ + sl.j0, sizeof(double) * (size_t)(sl.j1 - sl.j0),
                               cudaMemcpyDeviceToHost, d->copy_stream));
      if (R)
        CUDA_TRY(cudaMemcpyAsync(R + sl.c0, d->dR + sl.c0, sizeof(double) * (size_t)(sl.c1 - sl.c0),
                                 cudaMemcpyDeviceToHost, d->copy_stream));
    }
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(d->copy_stream));
    CUDA_TRY(cudaStreamSynchronize(d->stream));
    return 0;
  }
  CUDA_TRY(cudaMemcpyAsync(d->dU, U, sizeof(double) * n, cudaMemcpyHostToDevice, d->stream));
  if (Ut) CUDA_TRY(cudaMemcpyAsync(d->dUt, Ut, sizeof(double) * n, cudaMemcpyHostToDevice, d->stream));
  int ierr = device_eval(t, form, time, d->dU, Ut ? d->dUt : nullptr, shift, R ? d->dR : nullptr, J ? d->dJ : nullptr,
                         d->stream);
  if (ierr) return ierr;
  if (R) CUDA_TRY(cudaMemcpyAsync(R, d->dR, sizeof(double) * n, cudaMemcpyDeviceToHost, d->stream));
  if (J) CUDA_TRY(cudaMemcpyAsync(J, d->dJ, sizeof(double) * d->nnz, cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

// ---------------------------------------------------------------------------
// Evaluation without any device allocation of its own.
//
// The per-vertex partial sums (J_v, R_v) normally live in scratch that
// TDySetup allocates for the handle.  This variant takes them from a fixed
// array compiled into the library instead, so nothing in it allocates device
// memory.  The array is 64 MiB of doubles; every GPU that loads the library
// holds it until the process exits.  Host code never uses the array's name as
// an address (on the host it is only a stand-in for the symbol): the device
// address is looked up with cudaGetSymbolAddress once per device, while that
// device is current, by TDySetup (noalloc_resolve), so the call itself loads
// no module and allocates nothing, even the first time.
//
// All calls share the array and it keeps the last call's contents.  Nothing
// has to start at zero: vertex_kernel writes every partial that cell_kernel
// then reads in the same call.  Calls that overlap on the GPU (two streams, or
// two handles at once) race on the array and must be serialised by the caller.
#define TDY_NOALLOC_SCRATCH_DOUBLES (8ull << 20)
static __device__ __align__(256) double g_noalloc_scratch[TDY_NOALLOC_SCRATCH_DOUBLES];
static double *g_noalloc_ptr[kMaxDevices] = {};

static int noalloc_resolve(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return set_error(TDY_ERR_SUP, "device ordinal %d not supported", dev);
  std::lock_guard<std::mutex> lk(g_dev_mutex);
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_ptr[dev] = (double *)p;
  }
  return 0;
}

int device_eval_noalloc(_p_TDy *t, const double *dU, double *dR, double *dJ, void *stream) {
  DeviceState *d = t->dev;
  const long long need = t->setup.scratch_size;
  if (need > (long long)TDY_NOALLOC_SCRATCH_DOUBLES)
    return set_error(TDY_ERR_ARG_OUTOFRANGE,
                     "mesh needs %lld doubles of partial-sum scratch; the static scratch holds %llu (64 MiB). "
                     "Use TDyMPFAOSNESFunctionJacobianDevice for meshes this large",
                     need, (unsigned long long)TDY_NOALLOC_SCRATCH_DOUBLES);
  if (!(t->dtime > 0.0)) return set_error(TDY_ERR_USER, "SNES form needs TDySetDtimeForSNESSolver before evaluation");
  int dev = -1;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev != d->device)
    return set_error(TDY_ERR_USER, "current CUDA device %d is not the device %d this handle was set up on", dev,
                     d->device);
  double *scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_dev_mutex);
    scratch = g_noalloc_ptr[dev];  // resolved by TDySetup on this device
  }
  if (!scratch) return set_error(TDY_ERR_LIB, "static scratch address of device %d was not resolved at set-up", dev);
  cudaStream_t st = stream ? (cudaStream_t)stream : d->stream;
  DevArgs a = d->a;
  a.form = FORM_SNES;
  a.U = dU;
  a.Ut = nullptr;
  a.dt = t->dtime;
  a.shift = 1.0 / t->dtime;
  a.needR = dR != nullptr;
  a.needJ = dJ != nullptr;
  a.R = dR;
  a.J = dJ;
  a.scratch = scratch;
  int ierr = launch_eval(a, st, nullptr);
  if (ierr) return ierr;
  CUDA_TRY(cudaEventRecord(d->noalloc_ev, st));
  return 0;
}

int device_launches_per_eval(_p_TDy *t) {
  const DevArgs &a = t->dev->a;
  const int nvert = a.gen_apart ? 1 + (a.nC > 0) : (a.nC + a.ngen) > 0;
  const int ncell = (a.ngc > 0) + (a.nS > 0);
  return 1 + nvert + ncell;
}

int device_synchronize(_p_TDy *t) {
  CUDA_TRY(cudaStreamSynchronize(t->dev->stream));
  return 0;
}

int device_update_state_host(_p_TDy *t, const double *U) {
  DeviceState *d = t->dev;
  CUDA_TRY(cudaMemcpyAsync(d->dU, U, sizeof(double) * t->mesh.nc, cudaMemcpyHostToDevice, d->stream));
  DevArgs a = d->a;
  a.U = d->dU;
  diag_kernel<<<nblocks(a.nc, 256), 256, 0, d->stream>>>(a, d->diagS, d->diagMass);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  return 0;
}

int device_get_diagnostic(_p_TDy *t, int which, double *out) {
  DeviceState *d = t->dev;
  CUDA_TRY(cudaMemcpy(out, which == 0 ? d->diagS : d->diagMass, sizeof(double) * t->mesh.nc, cudaMemcpyDeviceToHost));
  return 0;
}

}  // namespace tdy
