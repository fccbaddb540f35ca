// Device code of the fused batched GGA forward and reduced implicit adjoint
// for sm_100a.  Included by the kernel-instance sources (wds_k_*.cu), each of
// which instantiates one kernel kind in one factor precision, so that the
// instances compile in parallel; the launchers (wds_launch.cu) reach them
// through the kernel selectors at the end of this file.
//
// A CTA holds `GR` independent scenario groups of 256 threads.  Each group owns
// one scenario at a time: its link conductances, the LDL^T factor of the node
// matrix and the node vectors live in shared memory (its link flows in L2) from
// the first Newton iteration to the terminal factorisation, so there is no host
// round trip inside the loop.  A network too large for that runs one scenario
// per CTA of 1024 threads, its state in shared memory as far as it fits.  The symbolic schedule (update lists, row and column
// structure, incidence lists) is staged once per CTA into shared memory as
// 16-bit tables and shared by the groups.  Groups synchronise on their own
// named barriers, so they advance independently.
//
// Per GGA iteration (dgga/solver.py:2922-3179):
//   link pass    P, Y from the headloss formulas and the link's term of the
//                right-hand side (one thread per link)
//   node pass    gather assembly of A (diagonal, pairs) and F in the
//                reference's scatter order; valve coefficients after the node
//                coefficients (a lane per valve, in valve order)
//   factor       left-looking LDL^T by elimination-tree level, the top levels
//                as one dense block inverted on the FP64 tensor cores
//   solve        forward/backward substitution by level around the top block's
//                inverse + refinement against the matrix-free operator A x
//   update       dq = Y - P dh, emitter update, relerr reduction, status
//                machine (valve status every iteration, link status on the
//                converged / periodic branches, per-scenario nextcheck)
// Implicit mode then runs the reduced Newton polish with Woodbury row
// replacement for ACTIVE PRVs (dgga/autodiff.py:965-1104) and stores the
// terminal factor and coefficients for the adjoint kernel.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <algorithm>
#include <type_traits>

#include "wds_internal.h"
#include "wds_math.cuh"

namespace wds {
namespace {

constexpr double kINF = __builtin_huge_val();
constexpr double kNaN = __builtin_nan("");
// A polish step keeps the factor in use while every link conductance P and
// emitter term of the step is within kReuseStep (relative) of the values it
// was factored with; the terminal state kept for the adjoint, within
// kReuseTerminal.
constexpr double kReuseStep = 1e-3;
constexpr double kReuseTerminal = 1e-4;
// ... and only once the previous step moved the flows by at most this
// fraction (sum |dq| / sum |q|): the polish is then in its quadratic regime,
// where a chord step equals the Newton step to rounding.
constexpr double kReuseFlow = 1e-6;

struct Sh {
  double *q, *P, *Y, *W, *V0, *V1, *V2, *hf, *xf, *red, *small;
  float* Wf;                      // the factor when it is kept in FP32 (W is then null)
  // per emitter slot: flow, coefficient, 1/hgrad, head loss, elevation (the
  // last two outside the state with n.ems = 0, see em_hloss)
  double *em_e, *em_ke, *em_emh, *em_hl, *em_el;
  int16_t* eslot;                 // [Nj] emitter slot of a junction or -1
  double* tb;                     // scratch of the top-block inversion (V2's storage)
  double* Mg;                     // [nT][top_ld(nT)] top-block inverse (shared memory when n.msm, else global)
  int *wcnt, *flag, *err;
  int8_t* S;
};

// View of the compact schedule tables.  Slot-valued tables (positions in the
// factor W, in the update-term list and in the row lists) hold Slot: uint16_t
// for networks whose tables fit 16 bits (staged into shared memory), uint32_t
// for large networks (tables read from global memory).  Junction, link and
// incidence indices are 16-bit in both.
template <class Slot>
struct TabT {
  static constexpr bool kWide = sizeof(Slot) == 4;
  const uint16_t* kf;         // [L] kind | flags << 8 (WDS_F_*, kStatusLink, kMinorLoss)
  const ValveRec* vrec;       // status-machine valves in the order of the valve pass
  // small networks: first term of the update list of every entry of L | its
  // diagonal flag << 15, one more at the end; the terms {slot L_ik, slot L_jk,
  // slot 1/D_k}
  const uint16_t* spair;
  const uint16_t* fpair;
  const Slot* colptr;         // [Nj+1]
  const uint16_t* rowidx;     // [nnzL]
  const uint16_t* levptr;     // [nlev+1] columns of a level (columns numbered in level order)
  const Slot* rptr;           // [Nj+1] row lists
  const uint32_t* rent;       // row entries slot | k << 16 (wide: 2 words, slot and k)
  const uint8_t* mfac;        // [nlev] mode: log2 G | wide << 7
  const uint8_t* mfwd;
  const uint8_t* mbwd;
  const uint16_t* inc_ptr;    // [Nj+1]
  const uint16_t* inc_split;  // [Nj]
  const uint16_t* inc;        // links at the junctions
  const int16_t* e1;          // [L] end codes
  const int16_t* e2;
  const uint16_t* pptr;       // [npairs+1]
  const uint16_t* plink;      // links of the pairs
  const Slot* pslot;          // [npairs]
  const Slot* fill;           // [nfill]
  // large networks (kWide): factor entries, their terms, column records of the
  // two substitutions, and the rounds of the factor and the substitutions (see factor_rounds)
  const uint4* act;
  const uint4* term;
  const uint4* colf;
  const uint4* colb;
  const uint2* frnd;
  const uint2* crnd;
  const uint2* brnd;
  const int* rptr3;           // [3][warps + 1] each warp's part of frnd, crnd, brnd
  const Slot* dslot;          // [nT (nT+1) / 2] slot of top-block entry (i >= j) or all ones

  // update list of the entry in `slot`: first term, term count, diagonal flag
  __device__ __forceinline__ void sp(int slot, int& pb, int& cnt, bool& diag) const {
    const int w = spair[slot], z = spair[slot + 1];
    pb = w & 0x7fff;
    cnt = (z & 0x7fff) - pb;
    diag = (w >> 15) != 0;
  }
  // row-list entry e: slot of L_jk and column k
  __device__ __forceinline__ void re(int e, int& slot, int& k) const {
    if constexpr (kWide) {
      const uint2 w = reinterpret_cast<const uint2*>(rent)[e];
      slot = (int)w.x;
      k = (int)w.y;
    } else {
      const uint32_t w = rent[e];
      slot = (int)(w & 0xffffu);
      k = (int)(w >> 16);
    }
  }
  __device__ __forceinline__ int cp(int j) const { return (int)colptr[j]; }
};
using STab = TabT<uint16_t>;
using LTab = TabT<uint32_t>;

template <class TB>
__device__ TB tab_view(const DevNet& n, const unsigned char* b) {
  using Slot = typename std::remove_pointer<decltype(TB::colptr)>::type;
  using S = typename std::remove_const<Slot>::type;
  TB t;
  t.kf = (const uint16_t*)(b + n.o_kf);
  t.vrec = (const ValveRec*)(b + n.o_vrec);
  t.spair = (const uint16_t*)(b + n.o_spair);
  t.fpair = (const uint16_t*)(b + n.o_fpair);
  t.colptr = (const S*)(b + n.o_colptr);
  t.rowidx = (const uint16_t*)(b + n.o_rowidx);
  t.levptr = (const uint16_t*)(b + n.o_levptr);
  t.rptr = (const S*)(b + n.o_rptr);
  t.rent = (const uint32_t*)(b + n.o_rent);
  t.mfac = (const uint8_t*)(b + n.o_mode);
  t.mfwd = t.mfac + n.nlev;
  t.mbwd = t.mfwd + n.nlev;
  t.inc_ptr = (const uint16_t*)(b + n.o_inc_ptr);
  t.inc_split = (const uint16_t*)(b + n.o_inc_split);
  t.inc = (const uint16_t*)(b + n.o_inc);
  t.e1 = (const int16_t*)(b + n.o_e1);
  t.e2 = (const int16_t*)(b + n.o_e2);
  t.pptr = (const uint16_t*)(b + n.o_pptr);
  t.plink = (const uint16_t*)(b + n.o_plink);
  t.pslot = (const S*)(b + n.o_pslot);
  t.fill = (const S*)(b + n.o_fill);
  t.dslot = (const S*)(b + n.o_dslot);
  if constexpr (TB::kWide) {
    t.act = (const uint4*)(b + n.o_act);
    t.term = (const uint4*)(b + n.o_term);
    t.colf = (const uint4*)(b + n.o_colf);
    t.colb = (const uint4*)(b + n.o_colb);
    t.frnd = (const uint2*)(b + n.o_frnd);
    t.crnd = (const uint2*)(b + n.o_crnd);
    t.brnd = (const uint2*)(b + n.o_brnd);
    t.rptr3 = (const int*)(b + n.o_rptr3);
  }
  return t;
}

// a link (kf: its entry of that table) whose coefficients the valve pass forms
__device__ __forceinline__ bool valve_link(uint32_t kf) {
  const int kd = (int)(kf & 0xff);
  return kd == WDS_KIND_PRV || kd == WDS_KIND_PSV || kd == WDS_KIND_FCV;
}

__device__ __forceinline__ double head_of(int c, const double* x, const double* hf) {
  return c >= 0 ? x[c] : hf[-c - 1];
}
__device__ __forceinline__ double junc_of(int c, const double* x) { return c >= 0 ? x[c] : 0.0; }

// ---------------------------------------------------------------- groups
// A group synchronises with its own named barrier (id 1 + group index).
template <int NT>
__device__ __forceinline__ int gtid() { return threadIdx.x & (NT - 1); }
// The warp of a group that runs the narrow levels: warp g mod 4 of group g,
// so that the co-resident groups' narrow chains issue from different SM
// sub-partitions (warp w of a CTA issues from sub-partition w mod 4).
template <int NT>
__device__ __forceinline__ bool in_narrow_warp() {
  constexpr int kWarps = NT / 32;
  const int g = (int)(threadIdx.x / NT) & 3;
  return (gtid<NT>() >> 5) == (g < kWarps ? g : 0);
}
template <int NT>
__device__ __forceinline__ void gsync() {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x / NT)), "r"(NT) : "memory");
}
template <int NT>
__device__ __forceinline__ bool gsync_or(bool p) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred ip, op;\n\tsetp.ne.u32 ip, %1, 0;\n\t"
      "bar.red.or.pred op, %2, %3, ip;\n\tselp.u32 %0, 1, 0, op;\n\t}"
      : "=r"(r)
      : "r"((unsigned)p), "r"(1 + (int)(threadIdx.x / NT)), "r"(NT)
      : "memory");
  return r != 0;
}

// Deterministic group sum of m <= 4 values (warp butterflies, then a fixed
// order over the warps); every thread gets the same result.
template <int NT>
__device__ void block_sum(double* v, int m, double* red) {
  for (int i = 0; i < m; ++i)
    for (int o = 16; o; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  const int w = gtid<NT>() >> 5, l = threadIdx.x & 31;
  gsync<NT>();
  if (l == 0)
    for (int i = 0; i < m; ++i) red[w * 4 + i] = v[i];
  gsync<NT>();
  for (int i = 0; i < m; ++i) {
    double s = 0.0;
    for (int ww = 0; ww < NT / 32; ++ww) s += red[ww * 4 + i];
    v[i] = s;
  }
}

// Group maximum of mx and minimum of mn (warp butterflies, then the warps'
// values in order); every thread gets both results.
template <int NT>
__device__ void block_maxmin(double& mx, double& mn, double* red) {
  for (int o = 16; o; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  const int w = gtid<NT>() >> 5, l = threadIdx.x & 31;
  gsync<NT>();
  if (l == 0) {
    red[w * 4] = mx;
    red[w * 4 + 1] = mn;
  }
  gsync<NT>();
  for (int ww = 0; ww < NT / 32; ++ww) {
    mx = fmax(mx, red[ww * 4]);
    mn = fmin(mn, red[ww * 4 + 1]);
  }
}

// ---------------------------------------------------------------- formulas
// emitterheadloss (dgga/solver.py:2368-2377)
__device__ __forceinline__ void emitter_hl(const DevNet& n, double e, double ke, double& hl,
                                           double& hg) {
  const double kea = fmax(ke, kCSMALL);
  const double ea = fmax(fabs(e), 1e-30);
  // (the default exponent 2 needs no power: pow_pos(x, 1) = x)
  hg = n.qexp * kea * (n.qexp == 2.0 ? ea : pow_pos(ea, n.qexp - 1.0));
  const bool lin = hg < n.rqtol;
  if (lin) hg = n.rqtol;
  hl = lin ? hg * e : hg * e / n.qexp;
}

// valvecoeff open branch (dgga/solver.py:2203-2219, :834-848)
__device__ __forceinline__ void valve_open(const DevNet& n, double q, double km, double& P,
                                           double& Y) {
  double hg = 2.0 * km * fabs(q);
  const bool lin = hg < n.rqtol;
  if (lin) hg = n.rqtol;
  const double hl = lin ? q * hg : q * hg / 2.0;
  if (km > 0.0) {
    P = 1.0 / hg;
    Y = hl / hg;
  } else {
    P = 1.0 / kCSMALL;
    Y = q;
  }
}

// pipecoeff, Hazen-Williams / Chezy-Manning (dgga/solver.py:2176-2201).  An
// infinite gradient gives P = 0, and with it or a head loss beyond the range of
// a double Y = NaN, as the plain divisions do (1 / inf, inf / inf): the scenario
// does not converge, and no pivot fails.
__device__ __forceinline__ void pipe_coef(const DevNet& n, double q, double r, double km,
                                          double& P, double& Y) {
  const double qa = fabs(q);
  double hg = n.hexp * r * pow_pos(fmax(qa, 1e-30), n.hexp - 1.0);
  const bool lin = hg < n.rqtol;
  if (lin) hg = n.rqtol;
  const double ex = lin ? 1.0 : n.hexp, rex = lin ? 1.0 : n.rhexp;  // hl = hg qa / ex
  if (km > 0.0) {
    const double hl = quotient(hg * qa, ex, rex) + km * qa * qa;
    hg = hg + 2.0 * km * qa;
    P = recip(hg);
    Y = copysign(quotient(hl, hg, P), q);
  } else {
    P = recip(hg);
    Y = quotient(q, ex, rex);
  }
  // by selects: a rare call instead costs the four-group kernel 7 %
  P = hg == kINF ? 0.0 : P;
  Y = hg * qa < kINF ? Y : kNaN;
}

// Pump parameters of one scenario: rows of [L] values read at pump links
// (the network's own, or the call's speed / pump_h0 / pump_r of
// implicit_solve, dgga/autodiff.py:1315-1342), read through the kernel
// arguments only where a pump needs them.  own_sp: the speeds are the call's,
// so the zero-speed and pumpstatus tests are taken from them instead of the
// network's link flags.
struct PumpTh {
  const FwdArgs& a;
  const DevNet& n;
  long long o;  // row offset of this scenario
  __device__ __forceinline__ bool own_sp() const { return a.th_sp != nullptr; }
  __device__ __forceinline__ double sp(int k) const { return a.th_sp ? a.th_sp[o + k] : n.pspeed[k]; }
  __device__ __forceinline__ double h0(int k) const { return a.th_h0 ? a.th_h0[o + k] : n.ph0[k]; }
  __device__ __forceinline__ double r(int k) const { return a.th_r ? a.th_r[o + k] : n.pr[k]; }
};

__device__ __forceinline__ PumpTh pump_th(const DevNet& n, const FwdArgs& a, int b) {
  return PumpTh{a, n, (long long)b * a.th_stride};
}

// A pump on the closed branch for its speed alone (hydcoeffs.c:696-701 via
// dgga/solver.py:673: setting == 0).
__device__ __forceinline__ bool zero_speed(const DevNet& n, const PumpTh& th, int k, int kd) {
  return th.own_sp() ? (kd == WDS_KIND_PUMP && th.sp(k) == 0.0)
                     : (n.flags[k] & WDS_F_ZERO_SPEED) != 0;
}

// pumpcoeff for every curve kind (dgga/solver.py:2221-2326)
__device__ void pump_coef(const DevNet& n, const PumpTh& th, int k, double q, double& P,
                          double& Y) {
  const int t = n.ptype[k];
  if (t == 3) {  // NOCURVE: an open valve
    P = 1.0 / kCSMALL;
    Y = q;
    return;
  }
  const double sgn = q < 0.0 ? -1.0 : 1.0;
  const double qa = q * sgn;
  const double spc = fmax(th.sp(k), 1e-12);
  double hg, hl;
  if (t == 2) {  // CUSTOM: piecewise-linear curve segment
    const int c0 = n.cptr[k], np = n.cptr[k + 1] - c0;
    const double* X = n.cx + c0;
    const double* Yc = n.cy + c0;
    const double qq = (fabs(q) / spc) * n.ucf_flow;
    int idx = 0;
    while (idx < np && X[idx] < qq) ++idx;
    const int k2 = min(max(idx, 1), np - 1), k1 = k2 - 1;
    double rc = (Yc[k2] - Yc[k1]) / (X[k2] - X[k1]);
    double h0c = Yc[k1] - rc * X[k1];
    h0c = h0c / n.ucf_head;
    rc = rc * n.ucf_flow / n.ucf_head;
    hg = (-rc) * spc;
    hl = (-h0c) * (spc * spc) + hg * q;
  } else {
    const double pn = n.pn[k];
    const double h0e = spc * spc * th.h0(k);
    const double re = th.r(k) * pow_pos(spc, 2.0 - pn);
    if (t == 0) {  // CONST_HP
      const double qac = fmax(qa, 1e-30);
      const double raw = -re / qac / qac;
      const bool big = raw > kCBIG, sml = raw < n.rqtol;
      hg = big ? kCBIG : (sml ? n.rqtol : raw);
      hl = (big || sml) ? -hg * q : re / (sgn * qac);
    } else if (pn == 1.0) {  // linear power function
      hg = re;
      hl = h0e + re * q;
    } else {  // power function; pow_pos(0, n-1) taken exactly
      const double nm1 = pn - 1.0;
      double pw;
      if (qa == 0.0)
        pw = nm1 > 0.0 ? 0.0 : ((nm1 < 0.0 && t == 1) ? kINF : 1.0);
      else
        pw = pow_pos(qa, nm1);
      const double raw = pn * re * pw;
      const bool sml = raw < n.rqtol;
      hg = sml ? n.rqtol : raw;
      hl = sml ? h0e + hg * q : h0e + hg * q / fmax(pn, 1e-30);
    }
  }
  P = 1.0 / hg;
  Y = hl / hg;
}

// Coefficients of a control valve that is not ACTIVE (valvecoeff, as
// restated in dgga/solver.py:862-903 and _valvecoeff_scalar): CLOSED is the
// 1/CBIG branch, otherwise the minor-loss Km (or 1/CSMALL for Km = 0).
__device__ __forceinline__ void valve_state_coef(const DevNet& n, double km, double qk, int sk,
                                                 double& P, double& Y) {
  const bool cl = sk <= WDS_CLOSED;
  double po, yo;
  if (km > 0.0) {
    double hg = 2.0 * km * fabs(qk);
    const bool lin = hg < n.rqtol;
    if (lin) hg = n.rqtol;
    const double hl = lin ? qk * hg : qk * hg / 2.0;
    po = 1.0 / hg;
    yo = hl / hg;
  } else {
    po = 1.0 / kCSMALL;
    yo = qk;
  }
  P = cl ? 1.0 / kCBIG : po;
  Y = cl ? qk : yo;
}

// PRV valve coefficients of one status-machine PRV (dgga/solver.py:862-903):
// returns pna (the non-ACTIVE P, zero when ACTIVE) and yna.
__device__ __forceinline__ void prv_open(const DevNet& n, int i, double qk, int sk, double& pna,
                                         double& yna) {
  double P;
  valve_state_coef(n, n.pcv_km[i], qk, sk, P, yna);
  pna = P * (sk == WDS_ACTIVE ? 0.0 : 1.0);
}

// Link coefficients of the headloss stage (dgga/solver.py:2923-2956).
// `adj` selects the adjoint/polish variant in which a status-machine PRV
// takes its valve coefficients directly (autodiff.py:838-847).
// `kf` is the link's entry of the table of that name.
__device__ __forceinline__ void link_coef(const DevNet& n, const PumpTh& th, int k, uint32_t kf,
                                          double q, int s, double r, bool adj, double& P,
                                          double& Y) {
  const int kd = (int)(kf & 0xff);
  if (kd == WDS_KIND_FCV) {  // the valve pass fills the GGA coefficients
    if (!adj) {
      P = 0.0;
      Y = 0.0;
    } else if (s == WDS_ACTIVE) {  // hloss = CBIG (q - qset), hgrad = CBIG
      P = 1.0 / kCBIG;
      Y = q - n.fcv_qs[n.link_fcv[k]];
    } else {
      valve_state_coef(n, n.fcv_km[n.link_fcv[k]], q, s, P, Y);
    }
    return;
  }
  if (kd == WDS_KIND_PRV || kd == WDS_KIND_PSV) {
    if (!adj) {
      P = 0.0;
      Y = 0.0;
    } else {
      double pna, yna;
      prv_open(n, n.link_pcv[k], q, s, pna, yna);
      P = pna;
      Y = (s == WDS_ACTIVE) ? q + 0.0 : yna;
    }
    return;
  }
  const bool still = th.own_sp() ? (kd == WDS_KIND_PUMP && th.sp(k) == 0.0)
                                 : (kf >> 8 & WDS_F_ZERO_SPEED) != 0;  // as zero_speed
  if (s <= WDS_CLOSED || still) {
    P = 1.0 / kCBIG;
    Y = q;
    return;
  }
  if (kd <= WDS_KIND_CVPIPE)
    pipe_coef(n, q, r, kf >> 8 & kMinorLoss ? n.km[k] : 0.0, P, Y);
  else if (kd == WDS_KIND_TCV)
    valve_open(n, q, n.km_tcv[k], P, Y);
  else if (kd == WDS_KIND_PRV_FIXED)
    valve_open(n, q, n.km[k], P, Y);
  else
    pump_coef(n, th, k, q, P, Y);
}

// d hloss / d(speed, H0, R) of one open pump at flow q with the curve
// segment / clamp branch frozen (dgga/autodiff.py:122-218, the CPU adjoint's
// pump theta; hydcoeffs.c:673-791).  Zero on the closed, zero-speed, NOCURVE
// and clamped constant-HP branches.
__device__ void pump_dtheta(const DevNet& n, const PumpTh& th, int k, double q, int st,
                            double& dw, double& dh0, double& dR) {
  dw = dh0 = dR = 0.0;
  const double w = th.sp(k);
  const int t = n.ptype[k];
  if (st <= WDS_CLOSED || w == 0.0 || t == 3) return;
  const double qa = fabs(q);
  if (t == 2) {  // CUSTOM: dw = 2 w H0c + Rc q on the frozen segment
    const int c0 = n.cptr[k], np = n.cptr[k + 1] - c0;
    const double* X = n.cx + c0;
    const double* Yc = n.cy + c0;
    const double spc = fmax(w, 1e-12);
    const double qq = (qa / spc) * n.ucf_flow;
    int idx = 0;
    while (idx < np && X[idx] < qq) ++idx;
    const int k2 = min(max(idx, 1), np - 1), k1 = k2 - 1;
    double rc = (Yc[k2] - Yc[k1]) / (X[k2] - X[k1]);
    double h0c = Yc[k1] - rc * X[k1];
    h0c = h0c / n.ucf_head;
    rc = rc * n.ucf_flow / n.ucf_head;
    dw = 2.0 * w * (-h0c) + (-rc) * q;
    return;
  }
  const double pn = n.pn[k], H0 = th.h0(k), R = th.r(k);
  if (t == 0) {  // CONST_HP: hloss = r / q on the unclamped branch only
    const double r = R * pow_pos(w, 2.0 - pn);
    const double hgr = qa > 0.0 ? -r / qa / qa : kINF;
    if (hgr > kCBIG || hgr < n.rqtol) return;
    dw = (2.0 - pn) * R * pow_pos(w, 1.0 - pn) / q;
    dR = pow_pos(w, 2.0 - pn) / q;
    return;
  }
  dh0 = w * w;
  if (pn == 1.0) {  // linear curve
    dw = 2.0 * w * H0 + R * q;
    dR = w * q;
    return;
  }
  const double nm1 = pn - 1.0;
  const double pw = qa == 0.0 ? (nm1 > 0.0 ? 0.0 : (nm1 < 0.0 ? kINF : 1.0)) : pow_pos(qa, nm1);
  const double hgr = pn * (R * pow_pos(w, 2.0 - pn)) * pw;
  if (hgr < n.rqtol) {  // RQtol clamp: hloss = h0 + RQtol q
    dw = 2.0 * w * H0;
    return;
  }
  dw = 2.0 * w * H0 + (2.0 - pn) * R * pow_pos(w, 1.0 - pn) * pw * q;
  dR = pow_pos(w, 2.0 - pn) * pw * q;
}

// ---------------------------------------------------------------- linear algebra
// Matrix-free (A x)_p of the node matrix: links with conductance P, emitter
// diagonal emh, CBIG on the downstream node of ACTIVE PRVs
// (dgga/autodiff.py:878-895; the same operator the forward assembles).
template <class TB>
__device__ __forceinline__ double amul_node(const DevNet& n, const TB& T, const Sh& s, int p,
                                            const double* x) {
  const double* P = s.P;
  const int8_t* S = s.S;
  double acc = 0.0;
  const int a = T.inc_ptr[p], m = T.inc_split[p], z = T.inc_ptr[p + 1];
  for (int e = a; e < m; ++e) {
    const int k = T.inc[e];
    acc += P[k] * (junc_of(T.e1[k], x) - junc_of(T.e2[k], x));
  }
  for (int e = m; e < z; ++e) {
    const int k = T.inc[e];
    acc += -(P[k] * (junc_of(T.e1[k], x) - junc_of(T.e2[k], x)));
  }
  const int es = s.eslot[p];
  acc = acc + (es >= 0 ? s.em_emh[es] : 0.0) * x[p];
  for (int c = n.npcv ? n.cb_ptr[p] : 0, ce = n.npcv ? n.cb_ptr[p + 1] : 0; c < ce; ++c) {
    const int i = n.cb_idx[c];
    const double act = S[n.pcv_link[i]] == WDS_ACTIVE ? 1.0 : 0.0;
    acc += x[p] * act * kCBIG;
  }
  return acc;
}

// Sum over a lane group of size 1 << lg (aligned groups inside a warp); every
// lane of the warp calls it with the same lg.
template <class FT>
__device__ __forceinline__ FT group_sum(FT v, int lg) {
  for (int o = (1 << lg) >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 1 / D of a pivot
__device__ __forceinline__ double inv_pivot(double w) { return recip(w); }
__device__ __forceinline__ float inv_pivot(float w) { return 1.0f / w; }

// The factor of the scenario in its storage precision FT (double, or float
// for the FP32 factor with FP64 refinement).
template <class FT>
__device__ __forceinline__ FT* wp(const Sh& s);
template <>
__device__ __forceinline__ double* wp<double>(const Sh& s) { return s.W; }
template <>
__device__ __forceinline__ float* wp<float>(const Sh& s) { return s.Wf; }

// Factor slots [t0, t1) (one level, or the Schur-complement step of the top
// block) on `nthr` threads (thread index t): the entries are split over lane
// groups of 1 << lg, each group reducing its entry's update list with warp
// shuffles.  Diagonal entries of factored columns become 1/D.
template <class TB, class FT>
__device__ __forceinline__ void fac_range(const TB& T, FT* W, int t0, int t1, int lg, int t,
                                          int nthr, bool& bad) {
  const int G = 1 << lg, li = t & (G - 1), per = nthr >> lg;
  for (int base = t0 + ((t & ~31) >> lg); base < t1; base += per) {  // a warp without items skips
    const int slot = base + ((t & 31) >> lg);
    const bool valid = slot < t1;
    bool diag = false;
    FT acc = 0;
    if (valid) {
      int pb, cnt;
      T.sp(slot, pb, cnt, diag);
      const int pe = pb + cnt;
      for (int pr = pb + li; pr < pe; pr += G) {
        const auto* f = T.fpair + 3 * pr;
        acc = fma(W[f[0]] * W[f[1]], W[f[2]], acc);
      }
    }
    acc = group_sum(acc, lg);
    if (valid && li == 0) {
      const FT w = W[slot] - acc;
      if (diag) {
        if (!(w > FT(0)) || !isfinite(w)) bad = true;
        W[slot] = inv_pivot(w);
      } else {
        W[slot] = w;
      }
    }
  }
}

// Forward substitution over rows [c0, c1): v_j = (v_j - sum_k L_jk D_k u_k) / D_j,
// or, for the rows of the top block (top), v_j = v_j - sum over the lower columns.
template <class TB, class FT>
__device__ __forceinline__ void fwd_range(const TB& T, const FT* W, double* v, int c0,
                                          int c1, int lg, int t, int nthr, bool top) {
  const int G = 1 << lg, li = t & (G - 1), per = nthr >> lg;
  for (int base = c0 + ((t & ~31) >> lg); base < c1; base += per) {
    const int j = base + ((t & 31) >> lg);
    const bool valid = j < c1;
    FT acc = 0;
    if (valid) {
      const int e1 = (int)T.rptr[j + 1];
      for (int e = (int)T.rptr[j] + li; e < e1; e += G) {
        int sl, k;
        T.re(e, sl, k);
        acc = fma(W[sl], (FT)v[k], acc);
      }
    }
    acc = group_sum(acc, lg);
    if (valid && li == 0) {
      const FT vj = (FT)v[j];
      v[j] = (double)(top ? vj - acc : (vj - acc) * W[T.colptr[j]]);
    }
  }
}

// One backward-substitution level, columns [c0, c1):
// x_j = u_j - (1/D_j) sum_i L_ij D_j x_i.
template <class TB, class FT>
__device__ __forceinline__ void bwd_level(const TB& T, const FT* W, double* v, int c0, int c1,
                                          int lg, int t, int nthr) {
  const int G = 1 << lg, li = t & (G - 1), per = nthr >> lg;
  for (int base = c0 + ((t & ~31) >> lg); base < c1; base += per) {
    const int j = base + ((t & 31) >> lg);
    const bool valid = j < c1;
    int cb = 0;
    FT acc = 0;
    if (valid) {
      cb = T.colptr[j];
      const int ce = T.colptr[j + 1];
      for (int e = cb + 1 + li; e < ce; e += G) acc = fma(W[e], (FT)v[T.rowidx[e]], acc);
    }
    acc = group_sum(acc, lg);
    if (valid && li == 0) v[j] = (double)fma(-W[cb], acc, (FT)v[j]);
  }
}

// 2^-h with h = ceil(e / 2) for x = m 2^e (m in [1, 2)), so that x 2^-2h lies
// in [0.5, 2); 1 for a diagonal that is not positive and finite (the pivot
// check then reports it).  Scaling by it is exact.
__device__ __forceinline__ double pow2_scale(double x) {
  if (!(x > 0.0) || !isfinite(x)) return 1.0;
  const long long e = ((__double_as_longlong(x) >> 52) & 0x7ff) - 1023;
  const long long h = (e + 1) >> 1;
  return __longlong_as_double((1023 - h) << 52);
}

// One double-precision tensor-core product: c += a b^T on an 8 x 8 tile, four
// columns deep (lane l holds a[l / 4][l % 4], b[l / 4][l % 4] and
// c[l / 4][2 (l % 4) + {0, 1}]).
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

constexpr int kTopTiles = WDS_TOP_MAX / 8;   // 8 x 8 tiles along one side
// One panel buffer of the inversion: the block's four columns [WDS_TOP_MAX][4],
// then the inverse of its 4 x 4 pivot block
constexpr int kTopPanel = 4 * WDS_TOP_MAX + 16;
// Doubles of group scratch: three panel buffers and the row scales
constexpr int kTopScratch = 3 * kTopPanel + WDS_TOP_MAX;

// The inversion's two barriers (ids beside the groups' own): the `warps` warps
// that hold tile rows hand a block's columns to the pivot warp (A) and take
// its inverse back (B).  The producers of either only arrive.
template <int NT>
__device__ __forceinline__ void top_arrive(int id, int warps) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id + (int)(threadIdx.x / NT)), "r"(32 * warps + 32)
               : "memory");
}
template <int NT>
__device__ __forceinline__ void top_wait(int id, int warps) {
  asm volatile("bar.sync %0, %1;" ::"r"(id + (int)(threadIdx.x / NT)), "r"(32 * warps + 32)
               : "memory");
}
constexpr int kTopA = 5, kTopB = 9;

// Inverse of the 4 x 4 pivot block at q (row-major), every lane the same (so
// that nothing is broadcast); lane 0 writes it to pin.  By its LDL^T, a
// reciprocal per pivot: pairs with one reciprocal (of a times the determinant)
// shorten the chain by 22 cycles each but leave 1.25 times the error in a solve
// on 960 systems of 7 to 45 junctions, and no case measurably faster.
__device__ __forceinline__ void top_pivot(const double* q, double* pin, int lane, int& bad) {
  const double a11 = q[0], a21 = q[4], a22 = q[5];
  const double i1 = recip(a11), l21 = a21 * i1;
  const double d22 = fma(-l21, a21, a22), i2 = recip(d22);
  const double a31 = q[8], l31 = a31 * i1;
  const double b32 = fma(-l31, a21, q[9]), l32 = b32 * i2;
  const double c33 = fma(-l32, b32, fma(-l31, a31, q[10]));
  const double a41 = q[12], l41 = a41 * i1;
  const double b42 = fma(-l41, a21, q[13]), l42 = b42 * i2;
  const double c43 = fma(-l42, b32, fma(-l41, a31, q[14]));
  const double c44 = fma(-l42, b42, fma(-l41, a41, q[15]));
  const double i3 = recip(c33), l43 = c43 * i3;
  const double d44 = fma(-l43, c43, c44), i4 = recip(d44);
  if (!(a11 > 0.0) || !(d22 > 0.0) || !(c33 > 0.0) || !(d44 > 0.0) || !isfinite(d22) ||
      !isfinite(d44))
    bad = 1;
  // rows of L^-1 (unit lower), then L^-T D^-1 L^-1 from its last row up
  const double m31 = fma(l32, l21, -l31), m42 = fma(l43, l32, -l42);
  const double m41 = -fma(l43, m31, fma(-l42, l21, l41));
  const double p43 = -l43 * i4, p42 = m42 * i4, p41 = m41 * i4;
  const double e32 = -l32 * i3, e31 = m31 * i3, e21 = -l21 * i2;
  const double p33 = fma(-l43, p43, i3), p32 = fma(-l43, p42, e32), p31 = fma(-l43, p41, e31);
  const double p22 = fma(m42, p42, fma(-l32, e32, i2));
  const double p21 = fma(m42, p41, fma(-l32, e31, e21));
  const double p11 = fma(m41, p41, fma(m31, e31, fma(-l21, e21, i1)));
  if (lane == 0) {
    double2* o = reinterpret_cast<double2*>(pin);
    o[0] = make_double2(p11, p21);
    o[1] = make_double2(p31, p41);
    o[2] = make_double2(p21, p22);
    o[3] = make_double2(p32, p42);
    o[4] = make_double2(p31, p32);
    o[5] = make_double2(p33, p43);
    o[6] = make_double2(p41, p42);
    o[7] = make_double2(p43, i4);
  }
}

// Publishes the four columns of block K from the tiles (their rows in every
// warp).
template <int K>
__device__ __forceinline__ void top_publish(int w, int lane, const double (&c)[kTopTiles][2],
                                            double* tb) {
  if (((lane & 3) >> 1) == (K & 1))
    *reinterpret_cast<double2*>(tb + (K % 3) * kTopPanel + (8 * w + (lane >> 2)) * 4 +
                                2 * (lane & 1)) = make_double2(c[K >> 1][0], c[K >> 1][1]);
}

// Block K of the inversion on a tile-row warp: every tile takes the block's
// rank-4 update, the tile that holds the next block's columns first, so that
// those go out (and the pivot warp inverts their pivot block) while the other
// tiles are still updated.
template <int NT, int K>
__device__ __forceinline__ void top_steps(int nT, int tiles, int w, int lane,
                                          double (&c)[kTopTiles][2], double* tb) {
  if constexpr (4 * K < WDS_TOP_MAX) {
    if (4 * K >= nT) return;
    constexpr int tK = K >> 1, tN = (K + 1) >> 1 < kTopTiles ? (K + 1) >> 1 : tK;
    const double* buf = tb + (K % 3) * kTopPanel;
    const double* pin = buf + 4 * WDS_TOP_MAX;
    const int i = lane >> 2, m = lane & 3;
    // this lane's row of its tile row (prow, when w == tK) and of tile tK's
    // columns lies in the pivot block, at (i % 4, m)
    const bool prow = (i >> 2) == (K & 1);
    const double one = prow && (i & 3) == m ? 1.0 : 0.0;
    top_wait<NT>(kTopB, tiles);
    const double2* u = reinterpret_cast<const double2*>(buf + (8 * w + i) * 4);
    const double2* pv = reinterpret_cast<const double2*>(pin + 4 * m);
    const double2 u0 = u[0], u1 = u[1], p0 = pv[0], p1 = pv[1];
    const double pim = pin[4 * (i & 3) + m];
    const double2 pk = *reinterpret_cast<const double2*>(pin + 4 * (i & 3) + 2 * (m & 1));
    double bN = buf[(8 * tN + i) * 4 + m];
    if (tN == tK) bN -= one;  // P - I
    // -T, T = U P^-1; its pivot rows are I - P^-1
    double a = -fma(u1.y, p1.y, fma(u1.x, p1.x, fma(u0.y, p0.y, u0.x * p0.x)));
    a = w == tK && prow ? pim - one : a;
    const bool own = w == tK && prow && (m >> 1) == (K & 1);  // holds -P^-1 afterwards
    auto tile = [&](int t, double b) {
      dmma(c[t], a, b);
      if (t == tK) {
        c[t][0] = own ? -pk.x : c[t][0];
        c[t][1] = own ? -pk.y : c[t][1];
      }
    };
    tile(tN, bN);
    if constexpr (4 * (K + 1) < WDS_TOP_MAX) {
      if (4 * (K + 1) < nT) {
        top_publish<K + 1>(w, lane, c, tb);
        top_arrive<NT>(kTopA, tiles);
      }
    }
#pragma unroll
    for (int t = 0; t < kTopTiles; ++t)
      if (t != tN && t < tiles) tile(t, buf[(8 * t + i) * 4 + m] - (t == tK ? one : 0.0));
    top_steps<NT, K + 1>(nT, tiles, w, lane, c, tb);
  }
}

// Inverse of the top block's Schur complement S (nT x nT, nT <= WDS_TOP_MAX)
// by symmetric block sweeps (Gauss-Jordan elimination without pivoting, four
// columns at a time in column order; the pivots of the 4 x 4 blocks are those
// of the LDL^T of S, so their signs are the positive-definiteness check).  S
// is first scaled to S' = D S D with D the power-of-two diagonal that brings
// diag(S') into [0.5, 2) (exact), and S^{-1} = D S'^{-1} D.
// Sweeping block k with pivot block P and columns U maps S_kk -> -P^-1,
// S_ik -> U_i P^-1 and S_ij -> S_ij - U_i P^-1 U_j^T; after all blocks the
// matrix is -S'^{-1}.  With P - I in the pivot rows of U the one rank-4 update
// gives the block's rows and columns as well: U - (U P^-1)(P - I) = U P^-1,
// without cancellation since the entries of P - I are at most about 2 after
// the scaling; only S_kk is then overwritten.
// Warp w holds tile row w (8 rows of the full matrix) in registers for all
// blocks, six 8 x 8 tiles, and each tile's update is one m8n8k4 FP64
// tensor-core product: a block costs a warp six of them and 4 FMAs per lane,
// where four single-column sweeps on 3 x 3 entries per thread cost 48
// multiplies and FMAs per lane and four barriers of the whole group.  A
// seventh warp inverts the pivot blocks (44 columns, alone / three groups per
// SM: 19.0 / 31.3 k cycles with the single-column sweeps, 11.2 / 16.8 k so with
// pivots in pairs, under 1 % more now).  What bounds it is the chain of a
// block: publish the columns, invert the 4 x 4 block (four reciprocals), read
// it back, update the next block's tile.  S is read from the factor slots
// listed in dslot, S^{-1} is written to Mg (row-major, rows of top_ld(nT)
// entries); tb: kTopScratch doubles of the group (a panel buffer is written
// again only when every warp is past its tiles two blocks before).  Returns 1
// when this thread saw a pivot that was not positive and finite.  Runs as a
// separate function so that its tiles do not add to the caller's registers.
template <int NT, class Slot, class FT>
__device__ __noinline__ int top_inverse(const FT* W, const Slot* dslot, double* tb,
                                        double* Mg, int nT) {
  static_assert(NT >= 4 * WDS_TOP_MAX + 32 && WDS_TOP_MAX % 8 == 0,
                "a warp per tile row and one for the pivots");
  const int w = gtid<NT>() >> 5, lane = threadIdx.x & 31, i = lane >> 2, m = lane & 3;
  const int tiles = (nT + 7) >> 3, r = 8 * w + i;
  // the pivot warp: 6 or 7, so that neighbouring groups' lie on different
  // SM sub-partitions
  const int wp = kTopTiles + ((int)(threadIdx.x / NT) & 1);
  if (w == wp) {
    int bad = 0;
    for (int k = 0, o = 0; 4 * k < nT; ++k, o = o == 2 * kTopPanel ? 0 : o + kTopPanel) {
      top_wait<NT>(kTopA, tiles);
      top_pivot(tb + o + 16 * k, tb + o + 4 * WDS_TOP_MAX, lane, bad);
      top_arrive<NT>(kTopB, tiles);
    }
    return bad;
  }
  if (w >= tiles) return 0;
  double c[kTopTiles][2];
#pragma unroll
  for (int t = 0; t < kTopTiles; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 8 * t + 2 * m + e;
      double x = r == j ? 1.0 : 0.0;  // rows beyond nT: identity
      if (r < nT && j < nT) {
        const int hi = r > j ? r : j, lo = r > j ? j : r;
        const Slot sl = dslot[hi * (hi + 1) / 2 + lo];
        x = sl != (Slot)~Slot(0) ? (double)W[sl] : 0.0;
      }
      c[t][e] = x;
    }
  double* sc = tb + 3 * kTopPanel;
#pragma unroll
  for (int t = 0; t < kTopTiles; ++t)
    if (t == w && m == (i >> 1)) sc[r] = pow2_scale((i & 1) ? c[t][1] : c[t][0]);
  asm volatile("bar.sync %0, %1;" ::"r"(kTopB + (int)(threadIdx.x / NT)), "r"(32 * tiles)
               : "memory");
  const double dr = sc[r];
#pragma unroll
  for (int t = 0; t < kTopTiles; ++t)
    if (t < tiles) {
      const double2 d = *reinterpret_cast<const double2*>(sc + 8 * t + 2 * m);
      c[t][0] *= dr * d.x;
      c[t][1] *= dr * d.y;
    }
  top_publish<0>(w, lane, c, tb);
  top_arrive<NT>(kTopA, tiles);
  top_steps<NT, 0>(nT, tiles, w, lane, c, tb);
  const int ld = top_ld(nT);
#pragma unroll
  for (int t = 0; t < kTopTiles; ++t)
    if (t < tiles) {
      const double2 d = *reinterpret_cast<const double2*>(sc + 8 * t + 2 * m);
      const int j = 8 * t + 2 * m;
      if (r < nT && j < nT)
        *reinterpret_cast<double2*>(Mg + r * ld + j) =
            make_double2(-c[t][0] * (dr * d.x), -c[t][1] * (dr * d.y));
    }
  return 0;
}

template <int NT>
__device__ __noinline__ void top_apply(const double* Mg, double* vT, int nT) {
  const int tid = gtid<NT>(), i = tid >> 2, li = tid & 3;
  double acc0 = 0.0, acc1 = 0.0;
  if (i < nT) {
    const double* row = Mg + i * top_ld(nT);
#pragma unroll
    for (int q = 0; q < WDS_TOP_MAX / 4; q += 2) {
      const int j0 = li + 4 * q, j1 = j0 + 4;
      if (j0 < nT) acc0 += row[j0] * vT[j0];
      if (j1 < nT) acc1 += row[j1] * vT[j1];
    }
  }
  double acc = group_sum(acc0 + acc1, 2);
  gsync<NT>();
  if (i < nT && li == 0) vT[i] = acc;
  gsync<NT>();
}

// Level-scheduled LDL^T.  Wide levels (many independent entries) use all the
// group's threads and a group barrier; narrow levels run on one warp alone,
// separated by __syncwarp.  W holds A on entry (pattern of L, fill zero) and
// on exit the unscaled columns L_ij D_j with 1/D_j in the diagonal slot, for
// the columns below the top block; the top block's slots hold its Schur
// complement and its inverse goes to s.Mg.  Returns true when every pivot was
// positive and finite.
template <int NT, class FT>
__device__ bool factor_rounds(const uint2* rec, const int* ptr, const uint4* ent,
                              const uint4* term, FT* W);
template <int NT, bool BACK, class FT>
__device__ void solve_rounds(const uint2* rec, const int* ptr, const uint4* cols, const uint2* rent,
                             const uint16_t* rowidx, const FT* W, double* v);

template <int NT, class FT, class TB>
__device__ bool factor(const DevNet& n, const TB& T, const Sh& s) {
  if constexpr (TB::kWide) {
    bool bad = factor_rounds<NT, FT>(T.frnd, T.rptr3, T.act, T.term, wp<FT>(s));
    if (n.nT > 0 && top_inverse<NT>((const FT*)wp<FT>(s), T.dslot, s.tb, s.Mg, n.nT)) bad = true;
    return !gsync_or<NT>(bad);
  } else {
  const int tid = gtid<NT>(), lane = tid & 31;
  const bool inw = in_narrow_warp<NT>();
  bool bad = false, prev_wide = true;
  // a level's mode and slot range are static: the next level's are loaded
  // while this level runs, so that a level starts with its own work
  int md_n = n.L0 > 0 ? T.mfac[0] : 0, t1_n = n.L0 > 0 ? T.colptr[T.levptr[1]] : 0;
  int t0 = 0;
  for (int lv = 0; lv < n.L0; ++lv) {
    const int md = md_n, t1 = t1_n;
    if (lv + 1 < n.L0) {
      md_n = T.mfac[lv + 1];
      t1_n = T.colptr[T.levptr[lv + 2]];
    }
    const bool wide = (md & 0x80) != 0;
    if (wide) {
      if (!prev_wide) gsync<NT>();
      fac_range(T, wp<FT>(s), t0, t1, md & 7, tid, NT, bad);
      gsync<NT>();
    } else if (inw) {
      fac_range(T, wp<FT>(s), t0, t1, md & 7, lane, 32, bad);
      __syncwarp();
    }
    prev_wide = wide;
    t0 = t1;
  }
  if (n.nT > 0) {
    // Schur complement of the top block: its slots minus the lower columns' updates
    const int md = T.mfac[n.L0];
    const int t0 = T.colptr[n.cT];
    if (!prev_wide) gsync<NT>();
    if (md & 0x80) fac_range(T, wp<FT>(s), t0, n.nnzL, md & 7, tid, NT, bad);
    else if (inw) fac_range(T, wp<FT>(s), t0, n.nnzL, md & 7, lane, 32, bad);
    gsync<NT>();
    if (top_inverse<NT>((const FT*)wp<FT>(s), T.dslot, s.tb, s.Mg, n.nT)) bad = true;
  }
  return !gsync_or<NT>(bad);
  }
}

// In-place (L D L^T) v = b: forward levels below the top block, the top rows'
// right-hand side, the dense top solve, backward levels below the top block.
template <int NT, class FT, class TB>
__device__ void solve(const DevNet& n, const TB& T, const Sh& s, double* v) {
  if constexpr (TB::kWide) {
    const uint2* re = reinterpret_cast<const uint2*>(T.rent);
    solve_rounds<NT, false, FT>(T.crnd, T.rptr3 + NT / 32 + 1, T.colf, re, T.rowidx, wp<FT>(s), v);
    if (n.nT > 0) top_apply<NT>(s.Mg, v + n.cT, n.nT);
    solve_rounds<NT, true, FT>(T.brnd, T.rptr3 + 2 * (NT / 32 + 1), T.colb, re, T.rowidx, wp<FT>(s), v);
    return;
  } else {
  const int tid = gtid<NT>(), lane = tid & 31;
  const bool inw = in_narrow_warp<NT>();
  bool prev_wide = true;
  // each level's mode and column range come from registers loaded a level ahead
  int md_n = n.L0 > 0 ? T.mfwd[0] : 0, c1_n = n.L0 > 0 ? T.levptr[1] : 0;
  int c0 = 0;
  for (int lv = 0; lv < n.L0; ++lv) {
    const int md = md_n, c1 = c1_n;
    if (lv + 1 < n.L0) {
      md_n = T.mfwd[lv + 1];
      c1_n = T.levptr[lv + 2];
    }
    const bool wide = (md & 0x80) != 0;
    if (wide) {
      if (!prev_wide) gsync<NT>();
      fwd_range(T, (const FT*)wp<FT>(s), v, c0, c1, md & 7, tid, NT, false);
      gsync<NT>();
    } else if (inw) {
      fwd_range(T, (const FT*)wp<FT>(s), v, c0, c1, md & 7, lane, 32, false);
      __syncwarp();
    }
    prev_wide = wide;
    c0 = c1;
  }
  if (n.nT > 0) {
    const int md = T.mfwd[n.L0];
    if (!prev_wide) gsync<NT>();
    if (md & 0x80) fwd_range(T, (const FT*)wp<FT>(s), v, n.cT, n.Nj, md & 7, tid, NT, true);
    else if (inw) fwd_range(T, (const FT*)wp<FT>(s), v, n.cT, n.Nj, md & 7, lane, 32, true);
    gsync<NT>();
    top_apply<NT>(s.Mg, v + n.cT, n.nT);
    prev_wide = true;
  }
  int mb_n = n.L0 > 0 ? T.mbwd[n.L0 - 1] : 0, b0_n = n.L0 > 0 ? T.levptr[n.L0 - 1] : 0;
  int b1 = n.L0 > 0 ? T.levptr[n.L0] : 0;
  for (int lv = n.L0 - 1; lv >= 0; --lv) {
    const int md = mb_n, b0 = b0_n;
    if (lv > 0) {
      mb_n = T.mbwd[lv - 1];
      b0_n = T.levptr[lv - 1];
    }
    const bool wide = (md & 0x80) != 0;
    if (wide) {
      if (!prev_wide) gsync<NT>();
      bwd_level(T, (const FT*)wp<FT>(s), v, b0, b1, md & 7, tid, NT);
      gsync<NT>();
    } else if (inw) {
      bwd_level(T, (const FT*)wp<FT>(s), v, b0, b1, md & 7, lane, 32);
      __syncwarp();
    }
    prev_wide = wide;
    b1 = b0;
  }
  gsync<NT>();
  }
}

// ---------------------------------------------------------------- large networks
// The levels of a large network read their tables from L2, and 32 warps walk
// every level, most of them without an item in the narrow upper ones.  Here a
// pass is one list of rounds per warp, holding only the rounds in which the
// warp has items (at most 32 >> lg), {first item, count | lg << 6 | top << 9 |
// barriers << 16}: the warp passes the group barriers that lie between its
// rounds (one between two levels unless one warp does both) and nothing else.
// The tables are read ahead: the record three rounds, the item's record two
// rounds, its first two terms per lane one round.  An item's sum is formed on
// 1 << lg lanes as in the routines above.
// Bound by issue and the L2 latency of lists longer than two entries a lane:
// solve and gradient of 33 scenarios of 3000 junctions 3.08 -> 2.43 ms, 64
// scenarios x 12 steps of 20 000 junctions 137 -> 111 ms (level loops over all
// warps before; with the level's lane groups instead of the round's 2.82 and
// 130 ms).

// Item of this lane in round r, or -1.
__device__ __forceinline__ int round_item(uint2 r) {
  const int i = (int)(threadIdx.x & 31) >> ((r.y >> 6) & 7);
  return i < (int)(r.y & 63u) ? (int)r.x + i : -1;
}

// The barriers before round r; rounds of one warp in a row need its own only.
template <int NT>
__device__ __forceinline__ void round_begin(uint2 r) {
  __syncwarp();
  for (int k = (int)(r.y >> 16); k > 0; --k) gsync<NT>();
}

// The LDL^T of the levels and the top block's Schur complement: ent holds
// {first term, count | diagonal << 31, slot, 0}, term {L_ik, L_jk, 1/D_k, 0}
// slots.  Returns whether a pivot was not positive and finite.
template <int NT, class FT>
__device__ __noinline__ bool factor_rounds(const uint2* rec, const int* ptr, const uint4* ent,
                                           const uint4* term, FT* W) {
  const uint2 none = make_uint2(0, 0);
  const uint4 nil = make_uint4(0, 0, 0, 0);
  const int w = gtid<NT>() >> 5, lane = threadIdx.x & 31, nr = ptr[w + 1] - ptr[w] - 1;
  rec += ptr[w];  // the list ends with the barriers after the last round
  bool bad = false;
  auto entry = [&](uint2 r) {
    const int i = round_item(r);
    return i >= 0 ? ent[i] : nil;
  };
  auto terms = [&](uint4 s, uint2 r, uint4& a, uint4& b) {
    const int l = (int)(r.y >> 6) & 7, li = lane & ((1 << l) - 1);
    const int cnt = (int)(s.y & 0x7fffffffu);
    a = li < cnt ? term[s.x + li] : nil;
    b = li + (1 << l) < cnt ? term[s.x + li + (1 << l)] : nil;
  };
  uint2 r0 = rec[0], r1 = nr > 0 ? rec[1] : none, r2 = nr > 1 ? rec[2] : none;
  uint4 s0 = entry(r0), s1 = entry(r1), a0, b0;
  terms(s0, r0, a0, b0);
  for (int i = 0; i < nr; ++i) {
    const uint2 r3 = i + 3 <= nr ? rec[i + 3] : none;
    const uint4 s2 = entry(r2);
    uint4 a1, b1;
    terms(s1, r1, a1, b1);
    round_begin<NT>(r0);
    const int lg = (int)(r0.y >> 6) & 7, G = 1 << lg, li = lane & (G - 1);
    const int cnt = (int)(s0.y & 0x7fffffffu);
    FT acc = 0;
    if (li < cnt) acc = fma(W[a0.x] * W[a0.y], W[a0.z], acc);
    if (li + G < cnt) acc = fma(W[b0.x] * W[b0.y], W[b0.z], acc);
    for (int e = li + 2 * G; e < cnt; e += G) {
      const uint4 f = term[s0.x + e];
      acc = fma(W[f.x] * W[f.y], W[f.z], acc);
    }
    acc = group_sum(acc, lg);
    if (round_item(r0) >= 0 && li == 0) {
      const FT x = W[s0.z] - acc;
      const bool diag = (s0.y >> 31) != 0;
      if (diag && (!(x > FT(0)) || !isfinite(x))) bad = true;
      W[s0.z] = diag ? inv_pivot(x) : x;
    }
    r0 = r1;
    r1 = r2;
    r2 = r3;
    s0 = s1;
    s1 = s2;
    a0 = a1;
    b0 = b1;
  }
  round_begin<NT>(r0);
  return bad;
}

// Forward substitution (BACK false: entries {slot, column} of the column's row)
// or backward substitution (BACK true: the column's own entries, rows in
// rowidx) in v; column records {first row entry, entries, diagonal slot, column}.
template <int NT, bool BACK, class FT>
__device__ __noinline__ void solve_rounds(const uint2* rec, const int* ptr, const uint4* cols,
                                          const uint2* rent, const uint16_t* rowidx,
                                          const FT* W, double* v) {
  const uint2 none = make_uint2(0, 0);
  const uint4 nil = make_uint4(0, 0, 0, 0);
  const int w = gtid<NT>() >> 5, lane = threadIdx.x & 31, nr = ptr[w + 1] - ptr[w] - 1;
  rec += ptr[w];
  auto column = [&](uint2 r) {
    const int j = round_item(r);
    return j >= 0 ? cols[j] : nil;
  };
  // entry e of the column: its slot and the index of its vector element
  auto entry = [&](uint4 c, int e, int& sl, int& k) {
    if constexpr (BACK) {
      sl = (int)c.z + 1 + e;
      k = rowidx[sl];
    } else {
      const uint2 x = rent[c.x + e];
      sl = (int)x.x;
      k = (int)x.y;
    }
  };
  auto first2 = [&](uint4 c, uint2 r, int& sa, int& ka, int& sb, int& kb) {
    const int l = (int)(r.y >> 6) & 7, li = lane & ((1 << l) - 1), n = (int)c.y;
    sa = ka = sb = kb = 0;
    if (li < n) entry(c, li, sa, ka);
    if (li + (1 << l) < n) entry(c, li + (1 << l), sb, kb);
  };
  uint2 r0 = rec[0], r1 = nr > 0 ? rec[1] : none, r2 = nr > 1 ? rec[2] : none;
  uint4 c0 = column(r0), c1 = column(r1);
  int sa, ka, sb, kb;
  first2(c0, r0, sa, ka, sb, kb);
  FT wa = W[sa], wb = W[sb], wd = W[c0.z];
  for (int i = 0; i < nr; ++i) {
    const uint2 r3 = i + 3 <= nr ? rec[i + 3] : none;
    const uint4 c2 = column(r2);
    int sa1, ka1, sb1, kb1;
    first2(c1, r1, sa1, ka1, sb1, kb1);
    round_begin<NT>(r0);
    const int lg = (int)(r0.y >> 6) & 7, G = 1 << lg, li = lane & (G - 1), n = (int)c0.y;
    FT acc = 0;
    if (li < n) acc = fma(wa, (FT)v[ka], acc);
    if (li + G < n) acc = fma(wb, (FT)v[kb], acc);
    for (int e = li + 2 * G; e < n; e += G) {
      int sl, k;
      entry(c0, e, sl, k);
      acc = fma(W[sl], (FT)v[k], acc);
    }
    acc = group_sum(acc, lg);
    if (round_item(r0) >= 0 && li == 0) {
      const int j = (int)c0.w;
      if constexpr (BACK) {
        v[j] = (double)fma(-wd, acc, (FT)v[j]);
      } else {
        const FT x = (FT)v[j] - acc;
        v[j] = (double)((r0.y >> 9) & 1u ? x : x * wd);
      }
    }
    wa = W[sa1];
    wb = W[sb1];
    wd = W[c1.z];
    ka = ka1;
    kb = kb1;
    r0 = r1;
    r1 = r2;
    r2 = r3;
    c0 = c1;
    c1 = c2;
  }
  round_begin<NT>(r0);
}

// x = A^{-1} rhs with `refine` refinement steps against the matrix-free A.
// unit >= 0 means rhs = e_unit.  An x outside shared memory (the Woodbury
// columns, refinement corrections and the unrolled adjoint in the global
// workspace, the solution of a large network) is solved in the temporary t
// when that lies inside, and stored, so that the substitutions chain on
// shared-memory latency.
template <int NT, class FT, class TB>
__device__ void solve_refined(const DevNet& n, const TB& T, const Sh& s, const double* rhs,
                              int unit, double* x, double* t, int refine) {
  const int tid = gtid<NT>();
  const bool via_t = !__isShared(x) && __isShared(t);
  double* v = via_t ? t : x;
  for (int p = tid; p < n.Nj; p += NT) v[p] = unit >= 0 ? (p == unit ? 1.0 : 0.0) : rhs[p];
  gsync<NT>();
  for (int it = 0;; ++it) {
    solve<NT, FT>(n, T, s, v);
    if (it > 0 || via_t) {
      for (int p = tid; p < n.Nj; p += NT) x[p] = it > 0 ? x[p] + v[p] : v[p];
      gsync<NT>();
    }
    if (it == refine) return;
    v = t;
    for (int p = tid; p < n.Nj; p += NT) {
      const double b = unit >= 0 ? (p == unit ? 1.0 : 0.0) : rhs[p];
      t[p] = b - amul_node(n, T, s, p, x);
    }
    gsync<NT>();
  }
}

// Small dense solve (Gaussian elimination, partial pivoting), one thread.
__device__ void dense_solve(double* C, double* y, int m) {
  for (int c = 0; c < m; ++c) {
    int piv = c;
    for (int r = c + 1; r < m; ++r)
      if (fabs(C[r * m + c]) > fabs(C[piv * m + c])) piv = r;
    if (piv != c) {
      for (int k = 0; k < m; ++k) {
        double tmp = C[c * m + k];
        C[c * m + k] = C[piv * m + k];
        C[piv * m + k] = tmp;
      }
      double tmp = y[c];
      y[c] = y[piv];
      y[piv] = tmp;
    }
    for (int r = c + 1; r < m; ++r) {
      const double f = C[r * m + c] / C[c * m + c];
      for (int k = c; k < m; ++k) C[r * m + k] -= f * C[c * m + k];
      y[r] -= f * y[c];
    }
  }
  for (int c = m - 1; c >= 0; --c) {
    double s = y[c];
    for (int k = c + 1; k < m; ++k) s -= C[c * m + k] * y[k];
    y[c] = s / C[c * m + c];
  }
}

// ---------------------------------------------------------------- assembly
// Head loss of emitter slot es and elevation of its junction p: in the state, or
// (n.ems = 0, where it has no room for them) the losses in hl, the scenario's row
// of hge that the terminal state takes over, the elevations in the network's
// table.  Shared and global loads by a branch that every thread takes alike: one
// pointer for both makes every load of the two generic (782 junctions, 16 384
// scenarios: 41.4 ms against 40.9).
__device__ __forceinline__ double em_hloss(const DevNet& n, const Sh& s, const double* hl, int es) {
  double v;
  if (n.ems) v = s.em_hl[es];
  else asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(hl + es));
  return v;
}
__device__ __forceinline__ double em_elev(const DevNet& n, const Sh& s, int p, int es) {
  double v;
  if (n.ems) v = s.em_el[es];
  else asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(n.el + p));
  return v;
}

// Headloss stage of a GGA iteration (dgga/solver.py:2923-2956): P and Y of every
// link, and 1/hgrad and head loss of every emitter.  What a link adds to the
// right-hand side at its ends is formed here too, once, into the solves'
// temporary: +Z at its first end and -Z at its second, Z = Y - q plus the
// grounding term P H of a fixed end (a link with one fixed end reaches one
// junction only); 0 for the control valves, which the valve pass adds.  The
// node pass then reads P and Z from shared memory where it used to gather q
// and Y from L2 and to test every incidence entry for valves and fixed ends (782
// junctions, three groups per SM: 18.5 -> 4.7 k cycles an iteration).
template <int NT, class TB>
__device__ void link_pass(const DevNet& n, const PumpTh& th, const TB& T, const Sh& s,
                          const double* rrow, double* hrow) {
  const int tid = gtid<NT>();
  double* Z = s.V2;
  // the next link's flow and resistance, in L2, are loaded while this link's
  // coefficients are formed
  int k = tid;
  double qn = k < n.L ? s.q[k] : 0.0, rn = k < n.L ? rrow[k] : 0.0;
  for (; k < n.L; k += NT) {
    const double qk = qn, rk = rn;
    const uint32_t kf = T.kf[k];
    const int kn = k + NT;
    if (kn < n.L) {
      qn = s.q[kn];
      rn = rrow[kn];
    }
    double P, Y;
    link_coef(n, th, k, kf, qk, s.S[k], rk, false, P, Y);
    s.P[k] = P;
    s.Y[k] = Y;
    const int c1 = T.e1[k], c2 = T.e2[k];
    double z = Y - qk;
    if (c2 < 0 && c1 >= 0) z += P * s.hf[-c2 - 1];
    if (c1 < 0 && c2 >= 0) z -= P * s.hf[-c1 - 1];
    Z[k] = valve_link(kf) ? 0.0 : z;
  }
  for (int es = tid; es < s.flag[2]; es += NT) {
    double hl, hg;
    emitter_hl(n, s.em_e[es], s.em_ke[es], hl, hg);
    if (n.ems) s.em_hl[es] = hl;
    else hrow[es] = hl;
    s.em_emh[es] = 1.0 / hg;
  }
}

// Assembly of the node matrix and right-hand side (linkcoeffs ->
// emittercoeffs -> nodecoeffs, solver.py:2958-3007) from the link pass, into W
// (pattern of L) and F = V0; Xflow saved for the junctions whose valves read it.
template <int NT, class FT, class TB>
__device__ void assemble_gga(const DevNet& n, const TB& T, const Sh& s, const double* dj,
                             const double* hrow) {
  const int tid = gtid<NT>();
  const double* Z = s.V2;
  for (int p = tid; p < n.Nj; p += NT) {
    const int a = T.inc_ptr[p], m = T.inc_split[p], z = T.inc_ptr[p + 1];
    const double dem = dj[p];  // (L2) requested before the incidence sums
    const int es = s.eslot[p];
    double dg = 0.0, F = 0.0;
    for (int e = a; e < z; ++e) {
      const int k = T.inc[e];
      dg += s.P[k];
      F += e < m ? Z[k] : -Z[k];
    }
    if (es >= 0) {
      const double emh = s.em_emh[es];
      dg = dg + emh;
      F = F + (em_hloss(n, s, hrow, es) + em_elev(n, s, p, es)) * emh - s.em_e[es];
    }
    wp<FT>(s)[T.colptr[p]] = (FT)dg;
    s.V0[p] = F - dem;
  }
  for (int i = NT - 1 - tid; i < n.nxf; i += NT) {  // flow excess of the held junctions
    const int p = n.xf_node[i], m = T.inc_split[p], z = T.inc_ptr[p + 1];
    double xf = 0.0;
    for (int e = T.inc_ptr[p]; e < z; ++e) {
      const int k = T.inc[e];
      const double q = valve_link(T.kf[k]) ? 0.0 : s.q[k];
      xf += e < m ? -q : q;
    }
    const int es = s.eslot[p];
    if (es >= 0) xf -= s.em_e[es];
    s.xf[i] = xf - dj[p];
  }
  for (int t = tid; t < n.npairs; t += NT) {
    double v = 0.0;
    for (int e = T.pptr[t]; e < T.pptr[t + 1]; ++e) v += -s.P[T.plink[e]];
    wp<FT>(s)[T.pslot[t]] = (FT)v;
  }
  for (int t = tid; t < n.nfill; t += NT) wp<FT>(s)[T.fill[t]] = FT(0);
  // valvecoeffs after nodecoeffs, in valve order: a lane of the last warp (the
  // fewest junctions) per valve loads its flow and status and forms its
  // coefficients before the barrier, all valves at once, and the lanes then
  // take their turns at what depends on the order (3 valves, three groups per
  // SM, with the status pass: 9.0 -> 6.0 k cycles an iteration against one
  // thread that took valve after valve).
  const int nv = n.npcv + n.nfcv, lane = threadIdx.x & 31;
  if (nv == 0) {
    gsync<NT>();
    return;
  }
  const bool mine = tid >= NT - 32;
  int o = 0, k = 0, j1 = 0, j2 = 0, off = 0, jc = 0, jo = 0, x1 = 0, x2 = 0;
  double qk = 0.0, pk = 0.0, yk = 0.0, set = 0.0, sg = 0.0;
  bool act = false;
  auto fetch = [&](int v) {
    const ValveRec& r = T.vrec[v];
    k = r.k;
    qk = s.q[k];
    o = r.fcv;
    j1 = r.j1;
    j2 = r.j2;
    off = r.off;
    x1 = r.x1;
    x2 = r.x2;
    jc = r.jc;
    jo = r.jo;
    set = r.set;
    sg = r.sgn;
    const int sk = s.S[k];
    act = sk == WDS_ACTIVE;
    if (o && act) {
      pk = 1.0 / kCBIG;
      yk = qk - set;
    } else {
      valve_state_coef(n, r.km, qk, sk, pk, yk);
      if (!o) pk = pk * (act ? 0.0 : 1.0);  // as prv_open
    }
  };
  if (mine && lane < nv) fetch(lane);
  gsync<NT>();
  if (mine) {
    FT* W = wp<FT>(s);
    for (int v = 0; v < nv; ++v) {
      if (v > 0 && (v & 31) == 0 && v + lane < nv) fetch(v + lane);
      if (lane == (v & 31)) {
        double dy = yk - qk;
        if (o) {  // FCV (fcvcoeff, hydcoeffs.c:1047-1097 as in dgga/solver.py:1665-1695)
          if (act) {  // the setting cuts the network: an outflow at n1, an inflow at n2
            if (x1 >= 0) s.xf[x1] -= set;
            if (x2 >= 0) s.xf[x2] += set;
            dy = -set;
          }
        } else {
          // prvcoeff / psvcoeff (hydcoeffs.c:959-1044 as in dgga/solver.py:
          // 862-903, 1647-1664): an ACTIVE valve holds the head of jc (PRV: n2,
          // PSV: n1) by a CBIG penalty and reads the flow excess there
          const double xfc = s.xf[x1];
          if (act) {
            dy = 0.0;
            W[T.colptr[jc]] += (FT)kCBIG;
            if (sg * xfc < 0.0) s.V0[jo] += xfc;
            s.V0[jc] += set * kCBIG;
            yk = qk + sg * xfc;
          }
        }
        W[off] += (FT)(-pk);
        W[T.colptr[j1]] += (FT)pk;
        W[T.colptr[j2]] += (FT)pk;
        s.V0[j1] += dy;
        s.V0[j2] -= dy;
        s.P[k] = pk;
        s.Y[k] = yk;
      }
      __syncwarp();
    }
  }
  gsync<NT>();
}

// Reduced-matrix assembly at the current state (dgga/autodiff.py:928-962):
// every link with its P, + emh diagonal, + CBIG on ACTIVE PRV downstream nodes.
template <int NT, class FT, class TB>
__device__ void assemble_reduced(const DevNet& n, const TB& T, const Sh& s) {
  const int tid = gtid<NT>();
  for (int p = tid; p < n.Nj; p += NT) {
    double dg = 0.0;
    for (int e = T.inc_ptr[p]; e < T.inc_ptr[p + 1]; ++e) dg += s.P[T.inc[e]];
    const int es = s.eslot[p];
    dg = dg + (es >= 0 ? s.em_emh[es] : 0.0);
    for (int c = n.npcv ? n.cb_ptr[p] : 0, ce = n.npcv ? n.cb_ptr[p + 1] : 0; c < ce; ++c) {
      const int i = n.cb_idx[c];
      dg += kCBIG * (s.S[n.pcv_link[i]] == WDS_ACTIVE ? 1.0 : 0.0);
    }
    wp<FT>(s)[T.colptr[p]] = (FT)dg;
  }
  for (int t = tid; t < n.npairs; t += NT) {
    double v = 0.0;
    for (int e = T.pptr[t]; e < T.pptr[t + 1]; ++e) v += -s.P[T.plink[e]];
    wp<FT>(s)[T.pslot[t]] = (FT)v;
  }
  for (int t = tid; t < n.nfill; t += NT) wp<FT>(s)[T.fill[t]] = FT(0);
  gsync<NT>();
}

// Coefficients at the current state for polish / terminal (autodiff.py:786-875):
// P, Y per link; emh per junction.
// With Pf / Ef (the P of every link and 1/hg of every emitter slot that the
// factor in use was formed with), `far` reports whether any of them moved
// by more than tol, relative; their loads are issued before the
// coefficients are formed.
template <int NT, class TB>
__device__ void adj_coeffs(const DevNet& n, const PumpTh& th, const TB& T, const Sh& s,
                           const double* rrow, double* hrow, const double* Pf = nullptr,
                           const double* Ef = nullptr, double tol = 0.0,
                           bool* far = nullptr) {
  const int tid = gtid<NT>();
  bool fr = false;
  int k = tid;
  double qn = 0.0, rn = 0.0, pn = 0.0;  // the next link's
  auto fetch = [&](int i) {
    qn = s.q[i];
    rn = rrow[i];
    pn = Pf ? Pf[i] : 0.0;
  };
  if (k < n.L) fetch(k);
  for (; k < n.L; k += NT) {
    const double qk = qn, rk = rn, p0 = pn;
    if (k + NT < n.L) fetch(k + NT);
    double P, Y;
    link_coef(n, th, k, T.kf[k], qk, s.S[k], rk, true, P, Y);
    s.P[k] = P;
    s.Y[k] = Y;
    if (Pf) fr = fr || !(fabs(P - p0) <= tol * fabs(p0));
  }
  const int nem = s.flag[2];
  for (int es = tid; es < nem; es += NT) {
    const double e0 = Ef ? Ef[es] : 0.0;
    double hl, hg;
    emitter_hl(n, s.em_e[es], s.em_ke[es], hl, hg);
    const double emh = 1.0 / hg;
    if (n.ems) s.em_hl[es] = hl;
    else hrow[es] = hl;
    s.em_emh[es] = emh;
    if (Ef) fr = fr || !(fabs(emh - e0) <= tol * fabs(e0));
  }
  if (far) *far = fr;
  gsync<NT>();
}

// Primal reduced Newton solve with ACTIVE control valves (the system of
// dgga/autodiff.py:965-1029): an ACTIVE valve fixes the head it holds
// (dH_jc = -r_valve) and frees its flow, which enters the balance rows as the
// column u = sgn (e_jc - e_jo) (sgn +1 for a PRV, jc = n2; -1 for a PSV,
// jc = n1).  With dH_jc known, the unknowns are the other heads and the valve
// flow in slot jc: M y = r', M = the factored A with column jc replaced by u
// (the transpose of the adjoint's row-replaced matrix), r' = rhs - A_red[:,jc]
// dH_jc.  Woodbury on the factor: A^{-1} u_a - e_jc (one solve per active
// valve, right-hand side e_jc - e_jo), C_ab = X_b[jc_a], and `outer`
// refinement steps against the true M (one on the last polish step)
// make the result independent of the unrefined inner solves.  Output: dH
// (with dH_jc = -r_valve) and the valve flow corrections dqv[p].  rhs: V0
// (kept).
template <int NT, class FT, class TB>
__device__ void primal_solve(const DevNet& n, const TB& T, const Sh& s, double* rp, double* dH,
                             double* res, double* sx, double* cols, const double* rprv,
                             bool any_act, int outer, bool cols_ready) {
  const double* rhs = s.V0;
  double* t = s.V2;
  const int tid = gtid<NT>();
  if (!any_act) {  // `outer` refinement steps (one on the last polish step)
    solve_refined<NT, FT>(n, T, s, rhs, -1, dH, t, outer);
    return;
  }
  const int p = n.npcv;
  double* C = s.small;             // p*p
  double* y = s.small + 4 * p * p; // p
  double* actf = y + 2 * p;        // p
  double* dqv = actf + p;          // p, output
  if (tid == 0)
    for (int i = 0; i < p; ++i) actf[i] = s.S[n.pcv_link[i]] == WDS_ACTIVE ? 1.0 : 0.0;
  for (int q = tid; q < n.Nj; q += NT) sx[q] = 0.0;
  gsync<NT>();
  if (tid == 0)
    for (int i = 0; i < p; ++i)
      if (actf[i] != 0.0) sx[n.pcv_jc[i]] = -rprv[i];
  gsync<NT>();
  // r' = rhs - A_red dH_fixed (A_red: the factored matrix without the valves' penalty)
  for (int q = tid; q < n.Nj; q += NT) {
    double acc = amul_node(n, T, s, q, sx);
    for (int c = n.cb_ptr[q]; c < n.cb_ptr[q + 1]; ++c)
      acc -= sx[q] * (s.S[n.pcv_link[n.cb_idx[c]]] == WDS_ACTIVE ? kCBIG : 0.0);
    rp[q] = rhs[q] - acc;
  }
  gsync<NT>();
  // the outer refinement below contracts the error of these unrefined solves
  solve_refined<NT, FT>(n, T, s, rp, -1, dH, t, 0);
  // the columns and C depend on the factor alone: a step that reuses the
  // previous step's factor reuses them too (cols_ready)
  for (int c = 0; c < (cols_ready ? 0 : p); ++c) {  // X_c = A^{-1} sgn_c (e_jc - e_jo); zero for inactive valves
    double* xc = cols + (size_t)c * n.Nj;
    if (actf[c] == 0.0) {
      for (int q = tid; q < n.Nj; q += NT) xc[q] = 0.0;
      gsync<NT>();
      continue;
    }
    for (int q = tid; q < n.Nj; q += NT) res[q] = 0.0;
    gsync<NT>();
    if (tid == 0) {
      res[n.pcv_jc[c]] = n.pcv_sgn[c];
      res[n.pcv_jo[c]] = -n.pcv_sgn[c];
    }
    gsync<NT>();
    solve_refined<NT, FT>(n, T, s, res, -1, xc, t, 0);
  }
  if (tid == 0 && !cols_ready)
    for (int a0 = 0; a0 < p; ++a0)
      for (int c = 0; c < p; ++c)
        C[a0 * p + c] = actf[a0] != 0.0 ? cols[(size_t)c * n.Nj + n.pcv_jc[a0]]
                                         : (a0 == c ? 1.0 : 0.0);
  gsync<NT>();
  // x <- x - sum_b z_b (X_b - e_jc_b),  z = C^{-1} (x[jc] act)
  auto wood = [&](double* x) {
    if (tid == 0) {
      double* Cc = C + p * p;  // working copy (the small buffer holds 4 p^2 for C)
      for (int i = 0; i < p * p; ++i) Cc[i] = C[i];
      for (int a0 = 0; a0 < p; ++a0) y[a0] = x[n.pcv_jc[a0]] * actf[a0];
      dense_solve(Cc, y, p);
    }
    gsync<NT>();
    for (int q = tid; q < n.Nj; q += NT) {
      double acc = 0.0;
      for (int c = 0; c < p; ++c) acc += cols[(size_t)c * n.Nj + q] * y[c];
      x[q] = x[q] - acc;
    }
    gsync<NT>();
    if (tid == 0)
      for (int c = 0; c < p; ++c) x[n.pcv_jc[c]] += y[c] * actf[c];
    gsync<NT>();
  };
  wood(dH);
  for (int it = 0; it < outer; ++it) {
    // res = r' - M y, M y = A y_z + sum_a u_a y_jc (y_z: y with the valve slots zero)
    for (int q = tid; q < n.Nj; q += NT) sx[q] = dH[q];
    gsync<NT>();
    if (tid == 0)
      for (int i = 0; i < p; ++i)
        if (actf[i] != 0.0) sx[n.pcv_jc[i]] = 0.0;
    gsync<NT>();
    for (int q = tid; q < n.Nj; q += NT) res[q] = rp[q] - amul_node(n, T, s, q, sx);
    gsync<NT>();
    if (tid == 0)
      for (int i = 0; i < p; ++i)
        if (actf[i] != 0.0) {
          const double v = n.pcv_sgn[i] * dH[n.pcv_jc[i]];
          res[n.pcv_jc[i]] -= v;
          res[n.pcv_jo[i]] += v;
        }
    gsync<NT>();
    solve_refined<NT, FT>(n, T, s, res, -1, sx, t, 0);
    wood(sx);
    for (int q = tid; q < n.Nj; q += NT) dH[q] = dH[q] + sx[q];
    gsync<NT>();
  }
  if (tid == 0)
    for (int i = 0; i < p; ++i) {
      dqv[i] = actf[i] != 0.0 ? dH[n.pcv_jc[i]] : 0.0;
      if (actf[i] != 0.0) dH[n.pcv_jc[i]] = -rprv[i];
    }
  gsync<NT>();
}

// doubles of V2: a node vector, a link vector (the link pass), or the top-block
// inversion's scratch
__host__ __device__ inline int v2_len(const DevNet& n) {
  const int m = n.Nj > n.L ? n.Nj : n.L;
  return n.nT > 0 && m < kTopScratch ? kTopScratch : m;
}

__host__ __device__ __forceinline__ size_t al16(size_t x) { return (x + 15) / 16 * 16; }

// The pieces of a scenario's state, in the order in which they claim shared
// memory on the large-network layout: first what is small or always in use,
// then the vector the substitutions run in, the solution, the factor, the
// conductances and the rest.  take(bytes) places a piece and returns its
// address (null when only sizes are wanted).
// On the small layout V1 follows V2, and with n.join V2 is a node vector that
// runs on into V1 where the link pass or the top block's inversion needs more:
// V1, the heads, is set by the solve after both (a network of more links than
// junctions then needs no more room for the link pass).
template <bool kWide, class Take>
__host__ __device__ __forceinline__ Sh place_state(const DevNet& n, Take&& take) {
  Sh s;
  s.q = nullptr;  // link flows and Y live in the global workspace (set by the kernel)
  s.Y = nullptr;
  s.red = (double*)take(8ull * 4 * 32);
  s.wcnt = (int*)take(4ull * 32);
  s.flag = (int*)take(16);      // [0] factor verdict, [1] error, [2] emitter count
  s.err = s.flag + 1;
  s.small = (double*)take(8ull * (4 * n.npcv * n.npcv + 5 * n.npcv + 8));
  s.hf = (double*)take(8ull * (n.Nf > 0 ? n.Nf : 1));
  s.xf = (double*)take(8ull * (n.nxf > 0 ? n.nxf : 1));
  s.em_e = (double*)take(8ull * n.emcap);
  s.em_ke = (double*)take(8ull * n.emcap);
  s.em_emh = (double*)take(8ull * n.emcap);
  s.em_hl = (double*)take(n.ems ? 8ull * n.emcap : 0);
  s.em_el = (double*)take(n.ems ? 8ull * n.emcap : 0);
  // the solves' temporary; idle while the matrix is factored, so the top
  // block's inversion works there
  const size_t jv = 8ull * n.Nj, lv = 8ull * v2_len(n);
  const bool join = !kWide && n.join;
  s.V2 = (double*)take(join ? jv : lv);
  s.tb = s.V2;
  if (!kWide) s.V1 = (double*)take(join && lv > al16(jv) + jv ? lv - al16(jv) : jv);
  // the top block's inverse, where it fits (else the kernel points it to the
  // scenario's slice of the global workspace)
  s.Mg = n.msm ? (double*)take(8ull * n.nT * top_ld(n.nT)) : nullptr;
  if (kWide) s.V1 = (double*)take(jv);
  if (n.fp32) {
    s.Wf = (float*)take(4ull * n.nnzL);
    s.W = nullptr;
  } else {
    s.W = (double*)take(8ull * n.nnzL);
    s.Wf = nullptr;
  }
  s.P = (double*)take(8ull * n.L);
  s.V0 = (double*)take(8ull * n.Nj);
  s.S = (int8_t*)take(n.L);
  s.eslot = (int16_t*)take(2ull * n.Nj);
  return s;
}

// The state at `base` (shared memory on the small-network layout).  The pieces
// lie at offsets the plan computed, kernel parameters: a piece's address is one
// addition wherever it is used, not a register held (or spilled) from the
// start of the scenario on (three groups: 372 -> 224 bytes of spill loads with
// the link pass of that time, 248 now; L1 beside 220 KB of shared memory does
// not hold the spills of 768 threads).
__device__ __forceinline__ Sh carve(const DevNet& n, unsigned char* base) {
  int i = 0;
  return place_state<false>(n, [&](size_t) { return base + n.so[i++]; });
}

// The state of the large-network layout: a piece in shared memory at `sm`, or
// (a negative offset) in the scenario's slice of the global workspace.
__device__ __forceinline__ Sh carve_split(const DevNet& n, unsigned char* sm,
                                          unsigned char* base) {
  int i = 0;
  return place_state<true>(n, [&](size_t) {
    const int o = n.so[i++];
    return o >= 0 ? sm + o : base + ~o;
  });
}

// The offsets of the state's pieces: one after the other; on the large-network
// layout each in the n.sm_state bytes of shared memory while they last, else in
// the global workspace.
void state_pieces(DevNet& n) {
  size_t os = 0, og = 0;
  int i = 0;
  auto take = [&](size_t bytes) -> unsigned char* {
    const bool in = !n.wide || os + al16(bytes) <= (size_t)n.sm_state;
    n.so[i++] = in ? (int)os : ~(int)og;
    (in ? os : og) += al16(bytes);
    return nullptr;
  };
  if (n.wide) place_state<true>(n, take);
  else place_state<false>(n, take);
  n.gstate = (int)((og + 255) / 256 * 256);
}

// Bytes of a scenario's state.
size_t smem_bytes(const DevNet& n) {
  size_t o = 0;
  auto take = [&](size_t bytes) -> unsigned char* {
    o += al16(bytes);
    return nullptr;
  };
  if (n.wide) place_state<true>(n, take);
  else place_state<false>(n, take);
  return o;
}

// Compact the scenario's emitters (junctions with a positive coefficient, as
// given by val[jnode[p]] > 0) into slots in increasing elimination order:
// eslot[p] = slot or -1, em_ke = coefficient, em_e = initial flow 1.0
// (hydraul.c initial EmitterFlow).  Returns false when they exceed emcap.
template <int NT>
__device__ bool build_emitters(const DevNet& n, const Sh& s, const double* val, int stride_node) {
  const int tid = gtid<NT>(), lane = threadIdx.x & 31, warp = tid >> 5;
  int total = 0;
  bool over = false;
  for (int base = 0; base < n.Nj; base += NT) {
    const int p = base + tid;
    double v = 0.0;
    if (p < n.Nj) v = val[stride_node ? n.jnode[p] : p];
    const bool em = p < n.Nj && v > 0.0;
    const unsigned mask = __ballot_sync(0xffffffffu, em);
    if (lane == 0) s.wcnt[warp] = __popc(mask);
    gsync<NT>();
    int off = total, sum = 0;
    for (int w = 0; w < NT / 32; ++w) {
      if (w < warp) off += s.wcnt[w];
      sum += s.wcnt[w];
    }
    const int slot = off + __popc(mask & ((1u << lane) - 1u));
    if (p < n.Nj) {
      if (em && slot < n.emcap) {
        s.eslot[p] = (int16_t)slot;
        s.em_ke[slot] = v;
        s.em_e[slot] = 1.0;
        s.em_emh[slot] = 0.0;
        if (n.ems) s.em_el[slot] = n.el[p];
      } else {
        s.eslot[p] = -1;
        if (em) over = true;
      }
    }
    total += sum;
    gsync<NT>();
  }
  if (tid == 0) s.flag[2] = total < n.emcap ? total : n.emcap;
  if (tid == 0) *s.err = 0;
  return !gsync_or<NT>(over);
}

// ---------------------------------------------------------------- CTA scenario rounds
// The CTAs of a launch are persistent: CTA `blk` of the `nblk` that run a plan
// holds `groups` scenario groups of NT threads (groups beyond it, in a CTA
// with more threads, stay idle), and group g takes scenario
// b = (r * groups + g) * nblk + blk in rounds r = 0, 1, ... while b < B.  The
// first nblk scenarios of a round go to group 0 of every CTA, so a partial
// last round runs one group per SM instead of filling a few CTAs, and a group
// with fewer co-resident groups runs faster (the kernels are latency-bound).
// The schedule tables are staged into shared memory once per CTA; a group's
// scenario state is its own slice of shared memory (global memory, per
// scenario, on the large-network layout), reused from round to round behind a
// group barrier.  `one(T, s, b)` solves scenario b.
template <int NT, class TB, class One>
__device__ __forceinline__ void cta_rounds(const DevNet& n, const DevWork& w, int B,
                                           int state_bytes, int blk, int nblk, int groups,
                                           One&& one, bool by_slot = false) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int g = threadIdx.x / NT;
  TB T;
  if constexpr (TB::kWide) {
    T = tab_view<TB>(n, (const unsigned char*)n.stab);
  } else {
    for (int i = threadIdx.x; i < n.stab_bytes / 16; i += blockDim.x)
      ((uint4*)smem_raw)[i] = n.stab[i];
    __syncthreads();
    T = tab_view<TB>(n, smem_raw);
  }
  if (g >= groups) return;  // a whole group; groups use their own barriers
  for (int r = 0;; ++r) {
    const long long bl = ((long long)r * groups + g) * nblk + blk;
    if (bl >= B) return;  // uniform per group
    const int b = (int)bl;
    if (r > 0) gsync<NT>();  // the previous scenario's last reads of the group state
    Sh s;
    if constexpr (TB::kWide)
      s = carve_split(n, smem_raw,
                      w.state + (size_t)(by_slot ? blk * groups + g : b) * n.gstate);
    else
      s = carve(n, smem_raw + n.stab_bytes + (size_t)g * state_bytes);
    one(T, s, b);
  }
}

// ---------------------------------------------------------------- forward kernel
// Forward of scenario b by one scenario group.
template <int NT, class TB, class FT>
__device__ __forceinline__ void forward_one(const DevNet& n, const DevWork& w, const FwdArgs& a,
                                            const TB& T, Sh s, int b) {
  s.q = w.lk + (size_t)b * 2 * n.L;
  s.Y = s.q + n.L;
  if (!n.msm) s.Mg = w.M + (size_t)b * n.nT * top_ld(n.nT);
  const double* rrow = a.r + (long long)b * a.r_stride;
  const double* kerow = a.ke + (long long)b * a.ke_stride;
  const double* drow = a.d + (long long)b * n.N;
  const double* rhrow = a.rh + (long long)b * n.N;
  const PumpTh th = pump_th(n, a, b);
  // the scenario's junction demands in elimination order, gathered once and
  // read coalesced by every assembly
  double* dj = w.dj + (size_t)b * n.Nj;
  for (int p = gtid<NT>(); p < n.Nj; p += NT) dj[p] = drow[n.jnode[p]];
  bool hf_nan = false;  // a reservoir/tank head that is NaN: nothing is solved
  for (int f = gtid<NT>(); f < n.Nf; f += NT) {
    const double h = rhrow[n.fnode[f]];
    hf_nan = hf_nan || isnan(h);
    s.hf[f] = h;
  }
  for (int k = gtid<NT>(); k < n.L; k += NT) {
    s.q[k] = a.q0 ? a.q0[(size_t)b * n.L + k] : n.q_init[k];
    s.S[k] = a.s0 ? a.s0[(size_t)b * n.L + k] : n.status0[k];
  }
  hf_nan = gsync_or<NT>(hf_nan);
  const bool em_ok = build_emitters<NT>(n, s, kerow, 1) && !hf_nan;
  if (a.e0) {  // warm start of the emitter flows (solver.py:2881-2887)
    for (int p = gtid<NT>(); p < n.Nj; p += NT) {
      const int es = s.eslot[p];
      if (es >= 0) s.em_e[es] = a.e0[(size_t)b * n.N + n.jnode[p]];
    }
    gsync<NT>();
  }
  const bool sm = a.sm != 0;
  const int maxtrials = sm ? a.max_iter + (n.extra_iter > 0 ? n.extra_iter : 0) : a.max_iter;
  int nextcheck = n.checkfreq;
  int iters = maxtrials + 1, info = WDS_INFO_UNCONVERGED;
  double relerr = 0.0;
  bool ran = false;
  const int rec_w = n.L + 2 * n.Nj;  // unrolled record: q [L], e [Nj], H [Nj] per iteration
  double* recb = a.rec ? a.rec + (size_t)b * maxtrials * rec_w : nullptr;
  for (int it = 1; it <= (em_ok ? maxtrials : 0); ++it) {
    if (recb) {  // state at the start of iteration it, for the unrolled reverse pass
      double* r = recb + (size_t)(it - 1) * rec_w;
      for (int k = gtid<NT>(); k < n.L; k += NT) r[k] = s.q[k];
      for (int p = gtid<NT>(); p < n.Nj; p += NT)
        r[n.L + p] = s.eslot[p] >= 0 ? s.em_e[s.eslot[p]] : 0.0;
    }
    // ---- headloss coefficients, assembly
    link_pass<NT>(n, th, T, s, rrow, w.hge + (size_t)b * n.Nj);
    gsync<NT>();
    assemble_gga<NT, FT>(n, T, s, dj, w.hge + (size_t)b * n.Nj);
    ran = true;
    if (!factor<NT, FT>(n, T, s)) {
      info = WDS_INFO_NOT_PD;
      iters = it;
      break;
    }
    // refinement only where it can matter for the convergence test (see
    // WdsForwardOpts.refine_band); relerr still holds the previous iteration's
    const bool refine_it = a.rband <= 0.0 || it > 20 || (it > 1 && relerr < a.rband);
    solve_refined<NT, FT>(n, T, s, s.V0, -1, s.V1, s.V2, refine_it ? a.refine : 0);
    if (recb) {
      double* r = recb + (size_t)(it - 1) * rec_w + n.L + n.Nj;
      for (int p = gtid<NT>(); p < n.Nj; p += NT) r[p] = s.V1[p];
    }
    // ---- newflows (hydsolver.c:358-514 as restated in solver.py:3092-3110)
    double sums[4] = {0.0, 0.0, 0.0, 0.0};
    {
      int k = gtid<NT>();
      double yn = k < n.L ? s.Y[k] : 0.0, qn = k < n.L ? s.q[k] : 0.0;  // next link's, from L2
      for (; k < n.L; k += NT) {
        const double yk = yn, qk = qn;
        const int kn = k + NT;
        if (kn < n.L) {
          yn = s.Y[kn];
          qn = s.q[kn];
        }
        const double dh = head_of(T.e1[k], s.V1, s.hf) - head_of(T.e2[k], s.V1, s.hf);
        double dq = yk - s.P[k] * dh;
        if ((T.kf[k] >> 8 & WDS_F_CHP) && dq > qk) dq = qk / 2.0;
        const double q2 = qk - dq;
        s.q[k] = q2;
        sums[0] += fabs(dq);
        sums[1] += fabs(q2);
      }
    }
    for (int p = gtid<NT>(); p < n.Nj; p += NT) {
      const int es = s.eslot[p];
      if (es >= 0) {
        const double hl = em_hloss(n, s, w.hge + (size_t)b * n.Nj, es);
        const double dqe = (hl - (s.V1[p] - em_elev(n, s, p, es))) * s.em_emh[es];
        const double en = s.em_e[es] - dqe;
        s.em_e[es] = en;
        sums[2] += fabs(dqe);
        sums[3] += fabs(en);
      }
    }
    // the first valve of this thread: its constants, before the reduction's barriers
    int vk = 0, vpsv = 0;
    double vhs = 0.0, vkm = 0.0;
    if (sm && gtid<NT>() < n.npcv) {
      const int i = gtid<NT>();
      vk = n.pcv_link[i];
      vhs = n.pcv_hset[i];
      vkm = n.pcv_km[i];
      vpsv = n.pcv_psv[i];
    }
    block_sum<NT>(sums, 4, s.red);
    const double dqsum = sums[0] + sums[2], qsum = sums[1] + sums[3];
    relerr = qsum > a.hacc ? dqsum / qsum : dqsum;
    if (!sm) {
      if (!recb && !(relerr > a.hacc)) {  // the unrolled map runs all its iterations
        iters = it;
        info = 0;
        break;
      }
      continue;
    }
    // ---- batched status machine (hydsolve, solver.py:3126-3179)
    bool vchg = false;
    for (int i = gtid<NT>(); i < n.npcv; i += NT) {
      if (i >= NT) {
        vk = n.pcv_link[i];
        vhs = n.pcv_hset[i];
        vkm = n.pcv_km[i];
        vpsv = n.pcv_psv[i];
      }
      const int k = vk;
      const double h1 = head_of(T.e1[k], s.V1, s.hf), h2 = head_of(T.e2[k], s.V1, s.hf);
      const double qk = s.q[k], hs = vhs, ht = n.htol;
      const int sk = s.S[k];
      const double hml = vkm * (qk * qk);
      const bool neg = qk < -n.qtol;
      int ns = sk;
      if (vpsv) {  // psvstatus (hydstatus.c:302-359 as in dgga/solver.py:1736-1765)
        if (sk == WDS_ACTIVE)
          ns = neg ? WDS_CLOSED : (h2 + hml > hs + ht ? WDS_OPEN : WDS_ACTIVE);
        else if (sk == WDS_OPEN)
          ns = neg ? WDS_CLOSED : (h1 < hs - ht ? WDS_ACTIVE : WDS_OPEN);
        else if (sk == WDS_CLOSED)
          ns = (h2 > hs + ht && h1 > h2 + ht) ? WDS_OPEN
               : ((h1 >= hs + ht && h1 > h2 + ht) ? WDS_ACTIVE : WDS_CLOSED);
        else if (sk == WDS_XPRESSURE)
          ns = neg ? WDS_CLOSED : sk;
      } else if (sk == WDS_ACTIVE)
        ns = neg ? WDS_CLOSED : (h1 - hml < hs - ht ? WDS_OPEN : WDS_ACTIVE);
      else if (sk == WDS_OPEN)
        ns = neg ? WDS_CLOSED : (h2 >= hs + ht ? WDS_ACTIVE : WDS_OPEN);
      else if (sk == WDS_CLOSED)
        ns = (h1 >= hs + ht && h2 < hs - ht) ? WDS_ACTIVE
             : ((h1 < hs - ht && h1 > h2 + ht) ? WDS_OPEN : WDS_CLOSED);
      else if (sk == WDS_XPRESSURE)
        ns = neg ? WDS_CLOSED : sk;
      if (ns != sk) {
        vchg = true;
        if (a.schg)  // schedule record: the valve pass changed link k
          atomicOr(&a.schg[((size_t)b * maxtrials + (it - 1)) * ((n.L + 31) >> 5) + (k >> 5)],
                   1u << (k & 31));
      }
      s.S[k] = (int8_t)ns;
    }
    vchg = gsync_or<NT>(vchg);
    const bool conv = relerr <= a.hacc;
    const bool br_conv = conv && it <= a.max_iter;
    const bool br_per = !conv && it <= n.maxcheck && nextcheck == it;
    bool chg = false;
    if (br_conv || br_per) {
      for (int k = gtid<NT>(); k < n.L; k += NT) {
        const uint32_t kf = T.kf[k];
        const int st0 = s.S[k];
        int st = (st0 == WDS_XHEAD || st0 == WDS_TEMPCLOSED) ? WDS_OPEN : st0;
        if (!(kf >> 8 & kStatusLink) && st == st0) continue;  // no rule applies
        const double dh = head_of(T.e1[k], s.V1, s.hf) - head_of(T.e2[k], s.V1, s.hf);
        const double qk = s.q[k];
        if (n.kind[k] == WDS_KIND_CVPIPE) {  // cvstatus
          const bool rev = qk < -n.qtol;
          if (fabs(dh) > n.htol)
            st = (dh < -n.htol || rev) ? WDS_CLOSED : WDS_OPEN;
          else if (rev)
            st = WDS_CLOSED;
        }
        if (th.own_sp()) {  // pumpstatus at the call's speed (dgga/solver.py:673-679)
          const double w = th.sp(k);
          if (n.kind[k] == WDS_KIND_PUMP && w > 0.0 && st >= WDS_OPEN) {
            const double hmax = (n.flags[k] & WDS_F_CHP) ? kBIG : w * w * n.phunit[k];
            st = (-dh > hmax + n.htol) ? WDS_XHEAD : WDS_OPEN;
          }
        } else if ((n.flags[k] & WDS_F_PUMP_LIVE) && st >= WDS_OPEN) {  // pumpstatus
          st = (-dh > n.phmax[k] + n.htol) ? WDS_XHEAD : WDS_OPEN;
        }
        if (n.kind[k] == WDS_KIND_FCV) {
          // fcvstatus (hydstatus.c:362-398 as in dgga/solver.py:1816-1826,
          // 1875-1877), from the status before the reopening
          st = st0;
          if (dh < -n.htol || qk < -n.qtol)
            st = WDS_XFCV;
          else if (st0 == WDS_XFCV && qk >= n.fcv_qs[n.link_fcv[k]])
            st = WDS_ACTIVE;
        }
        const int t = n.link_tl[k];
        if (t >= 0) {  // tankstatus
          const bool live = st > WDS_CLOSED;
          const double ht = s.hf[n.tl_tank[t]];
          const double dht = ht - head_of(n.tl_other[t], s.V1, s.hf);
          const double qq = qk * n.tl_qsign[t];
          const uint8_t fl = n.tl_flags[t];
          const bool full = (ht >= n.tl_hmax[t] - n.htol) && !(fl & WDS_TL_OVERFLOW);
          const bool empty = ht <= n.tl_hmin[t] + n.htol;
          const bool big = fabs(dht) > n.htol;
          const bool cbig = (dht < -n.htol) || (qq < -n.qtol);
          const bool cl_open = big ? cbig : (qq < -n.qtol);   // cvstatus from OPEN
          const bool cl_closed = big ? cbig : true;           // cvstatus from CLOSED
          const bool cut_f = (fl & WDS_TL_IS_PUMP) ? (fl & WDS_TL_PUMP_IN) != 0 : cl_open;
          const bool cut_e = (fl & WDS_TL_IS_PUMP) ? (fl & WDS_TL_PUMP_OUT) != 0 : !cl_closed;
          if (live && ((full && cut_f) || (empty && cut_e))) st = WDS_TEMPCLOSED;
        }
        if (st != st0) {
          chg = true;
          if (a.schg)  // schedule record: link k changed in this check
            atomicOr(&a.schg[((size_t)b * maxtrials + (it - 1)) * ((n.L + 31) >> 5) + (k >> 5)],
                     1u << (k & 31));
        }
        s.S[k] = (int8_t)st;
      }
      chg = gsync_or<NT>(chg);
    }
    if (a.sflags && gtid<NT>() == 0)  // iteration it ran, and which link-status branch
      a.sflags[(size_t)b * maxtrials + (it - 1)] = 4 | (br_conv ? 1 : 0) | (br_per ? 2 : 0);
    const bool stat_change = br_conv && (chg || vchg);
    if (br_conv && stat_change) nextcheck = it + n.checkfreq;
    if (br_per) nextcheck += n.checkfreq;
    if (conv && (it > a.max_iter || !stat_change)) {
      iters = it;
      info = 0;
      break;
    }
  }
  if (recb && em_ok && info == WDS_INFO_UNCONVERGED) {  // K iterations done
    iters = maxtrials;
    info = 0;
  }
  gsync<NT>();
  // condition proxy (dgga/solver.py:3026-3032) of the last iteration's matrix:
  // its diagonal again from the last iteration's coefficients (P, 1/hgrad),
  // into V0, in the order of the assembly
  double dratio = 0.0;
  if (a.diag && n.npcv > 0 && ran) {
    double mx = 0.0, mn = kINF;
    for (int p = gtid<NT>(); p < n.Nj; p += NT) {
      double dg = 0.0;
      for (int e = T.inc_ptr[p]; e < T.inc_ptr[p + 1]; ++e) {
        const int k = T.inc[e];
        dg += valve_link(T.kf[k]) ? 0.0 : s.P[k];
      }
      if (s.eslot[p] >= 0) dg = dg + s.em_emh[s.eslot[p]];
      s.V0[p] = dg;
    }
    gsync<NT>();
    if (gtid<NT>() == 0)
      for (int v = 0; v < n.npcv + n.nfcv; ++v) {
        const int o = n.vord[v], f = -1 - o;
        const int k = o < 0 ? n.fcv_link[f] : n.pcv_link[o];
        s.V0[o < 0 ? n.fcv_j1[f] : n.pcv_j1[o]] += s.P[k];
        s.V0[o < 0 ? n.fcv_j2[f] : n.pcv_j2[o]] += s.P[k];
        if (o >= 0 && s.P[k] == 0.0) s.V0[n.pcv_jc[o]] += kCBIG;
      }
    gsync<NT>();
    for (int p = gtid<NT>(); p < n.Nj; p += NT) {
      const double dv = fabs(s.V0[p]);
      mx = fmax(mx, dv);
      mn = fmin(mn, dv);
    }
    block_maxmin<NT>(mx, mn, s.red);
    dratio = mx / fmax(mn, 1e-300);
  }
  // junction heads of the GGA solution stay in V1
  double* Hs = w.scr + (size_t)b * w.nscr * n.Nj;  // global copy of heads for the polish
  if (a.polish >= 0 && info == 0) {
    for (int p = gtid<NT>(); p < n.Nj; p += NT) Hs[p] = s.V1[p];
    gsync<NT>();
    double* rp = Hs + n.Nj;
    double* res = rp + n.Nj;
    double* sx = res + n.Nj;
    double* cols = sx + n.Nj;                          // 2p Woodbury columns
    // small buffer: C [4p^2], y [2p], actf [p], row1 [p], then r_prv [p]
    double* rprv = s.small + 4 * n.npcv * n.npcv + 4 * n.npcv;
    // Factor reuse: once the previous step moved the flows by at most
    // kReuseFlow, a step keeps the factor in use (and its Woodbury columns)
    // while every link conductance P and emitter term 1/hg of the step is
    // within kReuseStep, relative, of the values it was factored with (kept
    // in the workspace's P / emh rows until the terminal store).  The
    // Jacobian then differs from the factored one by at most that fraction
    // in every entry, so the step's correction differs from the Newton
    // correction by that fraction of itself, which in the quadratic regime
    // is below rounding; the last step's outer refinement runs against
    // the current operator.  The terminal state kept for the adjoint reuses
    // it within kReuseTerminal: every adjoint solve takes two refinement
    // steps against the terminal operator, which leave the cube of that
    // distance.
    double* Pf = w.P + (size_t)b * n.L;     // P of each link and 1/hg of each
    double* Ef = w.emh + (size_t)b * n.Nj;  // emitter slot of the factor in use
    bool have = false, reuse = false, settled = false;
    for (int step = 0; step <= a.polish; ++step) {
      bool far = false;
      const bool cand = have && settled;
      adj_coeffs<NT>(n, th, T, s, rrow, w.hge + (size_t)b * n.Nj, cand ? Pf : nullptr,
                     cand ? Ef : nullptr, step == a.polish ? kReuseTerminal : kReuseStep, &far);
      reuse = cand && !gsync_or<NT>(far);
      if (!reuse) {
        assemble_reduced<NT, FT>(n, T, s);
        if (!factor<NT, FT>(n, T, s)) {
          info = WDS_INFO_NOT_PD;
          break;
        }
        // each thread keeps the entries it compares (the same index mapping)
        for (int k = gtid<NT>(); k < n.L; k += NT) Pf[k] = s.P[k];
        for (int es = gtid<NT>(); es < s.flag[2]; es += NT) Ef[es] = s.em_emh[es];
        have = true;
      }
      if (step == a.polish) break;  // terminal factor: keep it
      // residuals (autodiff.py:1032-1050); r_l overwrites Y
      double yn = gtid<NT>() < n.L ? s.Y[gtid<NT>()] : 0.0;  // the next link's, from L2
      for (int k = gtid<NT>(); k < n.L; k += NT) {
        const double yk = yn;
        if (k + NT < n.L) yn = s.Y[k + NT];
        const double hl = s.P[k] != 0.0 ? yk / s.P[k] : 0.0;
        s.Y[k] = hl - (head_of(T.e1[k], Hs, s.hf) - head_of(T.e2[k], Hs, s.hf));
      }
      bool any_act = false;
      for (int i = gtid<NT>(); i < n.npcv; i += NT) {
        const bool act = s.S[n.pcv_link[i]] == WDS_ACTIVE;
        rprv[i] = (Hs[n.pcv_jc[i]] - n.pcv_hset[i]) * (act ? 1.0 : 0.0);
        any_act |= act;
      }
      any_act = gsync_or<NT>(any_act);
      for (int p = gtid<NT>(); p < n.Nj; p += NT) {
        const int a0 = T.inc_ptr[p], m = T.inc_split[p], z = T.inc_ptr[p + 1];
        double mm = 0.0, bt = 0.0;
        for (int e = m; e < z; ++e) {
          const int k = T.inc[e];
          mm += s.q[k];
          bt += s.P[k] * s.Y[k];
        }
        for (int e = a0; e < m; ++e) {
          const int k = T.inc[e];
          mm += -s.q[k];
          bt += -(s.P[k] * s.Y[k]);
        }
        const int es = s.eslot[p];
        double re = 0.0, emh = 0.0;
        if (es >= 0) {
          const double hl = em_hloss(n, s, w.hge + (size_t)b * n.Nj, es);
          re = hl - (Hs[p] - em_elev(n, s, p, es));
          mm = mm - s.em_e[es];
          emh = s.em_emh[es];
        }
        mm = mm - dj[p];
        s.V0[p] = (mm - bt) + emh * re;
      }
      gsync<NT>();
      // a Newton step corrects the rounding of the step before it: only the
      // last polish step's solve sets the final state, so it alone refines
      primal_solve<NT, FT>(n, T, s, rp, s.V1, res, sx, cols, rprv, any_act,
                           step == a.polish - 1 ? 1 : 0, reuse);
      // dq, de, state update
      double mv[2] = {0.0, 0.0};  // sum |dq|, sum |q|
      for (int k = gtid<NT>(); k < n.L; k += NT) {
        const double b1 = junc_of(T.e1[k], s.V1), b2 = junc_of(T.e2[k], s.V1);
        double dq = -s.P[k] * (s.Y[k] + (b2 - b1));
        const int i = n.link_pcv[k];
        if (i >= 0 && s.S[k] == WDS_ACTIVE)  // the free valve flow, solved in slot jc
          dq = s.small[4 * n.npcv * n.npcv + 3 * n.npcv + i];
        const double q2 = s.q[k] + dq;
        s.q[k] = q2;
        mv[0] += fabs(dq);
        mv[1] += fabs(q2);
      }
      for (int p = gtid<NT>(); p < n.Nj; p += NT) {
        const int es = s.eslot[p];
        if (es >= 0) {
          const double hl = em_hloss(n, s, w.hge + (size_t)b * n.Nj, es);
          const double re = hl - (Hs[p] - em_elev(n, s, p, es));
          s.em_e[es] = s.em_e[es] + (s.V1[p] - re) * s.em_emh[es];
        }
        Hs[p] = Hs[p] + s.V1[p];
      }
      block_sum<NT>(mv, 2, s.red);  // its barriers publish the updates above
      settled = mv[0] <= kReuseFlow * mv[1];
    }
    if (info == 0) {  // store the terminal state for the adjoint
      FT* Wt = reinterpret_cast<FT*>(w.W) + (size_t)b * n.nnzL;
      for (int t = gtid<NT>(); t < n.nnzL; t += NT) Wt[t] = wp<FT>(s)[t];
      if (n.msm && w.M) {
        double* Mt = w.M + (size_t)b * n.nT * top_ld(n.nT);
        for (int t = gtid<NT>(); t < n.nT * top_ld(n.nT); t += NT) Mt[t] = s.Mg[t];
      }
      for (int k = gtid<NT>(); k < n.L; k += NT) {
        const double q = s.q[k];
        w.P[(size_t)b * n.L + k] = s.P[k];
        double dr = 0.0;
        const int st = s.S[k];
        const bool closed = st <= WDS_CLOSED || zero_speed(n, th, k, n.kind[k]);
        if ((n.flags[k] & WDS_F_IS_PIPE) && !closed) {
          const double sgn = q < 0.0 ? -1.0 : 1.0, qa = q * sgn;
          const double pw = pow_pos(fmax(qa, 1e-30), n.hexp - 1.0);
          const double hgr = n.hexp * rrow[k] * pw;
          if (hgr >= n.rqtol) dr = (qa >= 1e-30 ? pw * qa : pow_any(qa, n.hexp)) * sgn;
        }
        w.dr[(size_t)b * n.L + k] = dr;
        const int ip = n.link_pump[k];
        if (ip >= 0) {
          double* dp = w.dpump + (size_t)b * 3 * n.npump;
          pump_dtheta(n, th, k, q, st, dp[ip], dp[n.npump + ip], dp[2 * n.npump + ip]);
        }
      }
      for (int p = gtid<NT>(); p < n.Nj; p += NT) {
        const int es = s.eslot[p];
        double hge = 1.0, dke = 0.0, emh = 0.0;
        if (es >= 0) {
          const double ke = s.em_ke[es], ee = s.em_e[es];
          double hl;
          emitter_hl(n, ee, ke, hl, hge);
          const double ea = fabs(ee);
          const double pw = pow_pos(fmax(ea, 1e-30), n.qexp - 1.0);
          const double raw = n.qexp * fmax(ke, kCSMALL) * pw;
          dke = (raw < n.rqtol || ke < kCSMALL) ? 0.0 : pw * ee;
          emh = s.em_emh[es];
        }
        w.emh[(size_t)b * n.Nj + p] = emh;
        w.hge[(size_t)b * n.Nj + p] = hge;
        w.dke[(size_t)b * n.Nj + p] = dke;
      }
      const int pc = n.npcv > 0 ? n.npcv : 1;
      for (int i = gtid<NT>(); i < n.npcv; i += NT)
        w.act[(size_t)b * pc + i] = s.S[n.pcv_link[i]] == WDS_ACTIVE ? 1 : 0;
    }
    for (int p = gtid<NT>(); p < n.Nj; p += NT) s.V1[p] = Hs[p];
    gsync<NT>();
  }
  gsync<NT>();
  if (hf_nan) info = WDS_INFO_BAD_HEAD;
  else if (!em_ok) info = WDS_INFO_EMITTER_CAP;
  if (gtid<NT>() == 0) w.valid[b] = (a.polish >= 0 && info == 0) ? 1 : 0;
  // ---- outputs
  double* hrow = a.head + (size_t)b * n.N;
  double* erow = a.emit + (size_t)b * n.N;
  for (int f = gtid<NT>(); f < n.Nf; f += NT) {
    hrow[n.fnode[f]] = s.hf[f];
    erow[n.fnode[f]] = 0.0;
  }
  for (int p = gtid<NT>(); p < n.Nj; p += NT) {
    const int nd = n.jnode[p];
    hrow[nd] = s.V1[p];
    const int es = s.eslot[p];
    erow[nd] = es >= 0 ? s.em_e[es] : 0.0;
  }
  for (int k = gtid<NT>(); k < n.L; k += NT) {
    a.flow[(size_t)b * n.L + k] = s.q[k];
    a.status[(size_t)b * n.L + k] = s.S[k];
  }
  if (gtid<NT>() == 0) {
    a.iters[b] = iters;
    a.relerr[b] = relerr;
    a.info[b] = info;
    if (a.diag) a.diag[b] = dratio;
  }
}

template <int NT, class TB, class FT>
__device__ __forceinline__ void forward_body(const DevNet& n, const DevWork& w, const FwdArgs& a,
                                             int state_bytes, int blk, int nblk, int groups) {
  cta_rounds<NT, TB>(n, w, a.B, state_bytes, blk, nblk, groups, [&](const TB& T, Sh s, int b) {
    forward_one<NT, TB, FT>(n, w, a, T, s, b);
  });
}

// ---------------------------------------------------------------- adjoint kernel
// Node adjoint with constraint rows (autodiff.py:1107-1154) and the
// theta contraction (autodiff.py:1246-1312).
// Adjoint of right-hand side b by one scenario group.
// With a.unit the right-hand side is the unit head adjoint of one node and only
// the resistance gradient is wanted.  `slot` numbers the scratch vectors.
template <int NT, class TB, class FT>
__device__ __forceinline__ void adjoint_one(const DevNet& n, const DevWork& w, const AdjArgs& a,
                                            const TB& T, Sh s, int b, int slot) {
  // kept state of scenario bf (several right-hand sides per scenario read the
  // same factor); right-hand sides, results and scratch are per b
  const int bf = (a.v0 + b) / (a.rhs_per > 1 ? a.rhs_per : 1);
  double* Mt = w.M + (size_t)bf * n.nT * top_ld(n.nT);  // terminal top-block inverse of the forward
  if (!w.valid[bf]) return;  // uniform per group
  if (n.msm)
    for (int t = gtid<NT>(); t < n.nT * top_ld(n.nT); t += NT) s.Mg[t] = Mt[t];
  else
    s.Mg = Mt;
  const FT* Wt = reinterpret_cast<const FT*>(w.W) + (size_t)bf * n.nnzL;
  for (int t = gtid<NT>(); t < n.nnzL; t += NT) wp<FT>(s)[t] = Wt[t];
  for (int k = gtid<NT>(); k < n.L; k += NT) s.P[k] = w.P[(size_t)bf * n.L + k];
  const int pc = n.npcv > 0 ? n.npcv : 1;
  // status is only consulted for ACTIVE flags of PRVs
  for (int k = gtid<NT>(); k < n.L; k += NT) {
    const int i = n.link_pcv[k];
    s.S[k] = (i >= 0 && w.act[(size_t)bf * pc + i]) ? WDS_ACTIVE : WDS_OPEN;
  }
  gsync<NT>();
  // emitter slots from the stored 1/hgrad (positive exactly at emitters)
  build_emitters<NT>(n, s, w.emh + (size_t)bf * n.Nj, 0);
  for (int p = gtid<NT>(); p < n.Nj; p += NT) {
    const int es = s.eslot[p];
    if (es >= 0) s.em_emh[es] = w.emh[(size_t)bf * n.Nj + p];
  }
  gsync<NT>();
  const bool unit = a.unit != nullptr;
  const int unode = unit ? a.unit[(a.v0 + b) % a.rhs_per] : -1;
  const double* gH = unit ? nullptr : a.gH + (size_t)b * n.N;
  const double* gQ = unit ? nullptr : a.gQ + (size_t)b * n.L;
  const double* gE = unit ? nullptr : a.gE + (size_t)b * n.N;
  // r = B^T P gQ - em gE / hge - gH
  if (unit)
    for (int p = gtid<NT>(); p < n.Nj; p += NT) s.V0[p] = n.jnode[p] == unode ? -1.0 : 0.0;
  else for (int p = gtid<NT>(); p < n.Nj; p += NT) {
    const int a0 = T.inc_ptr[p], m = T.inc_split[p], z = T.inc_ptr[p + 1];
    double acc = 0.0;
    for (int e = m; e < z; ++e) {
      const int k = T.inc[e];
      acc += s.P[k] * gQ[k];
    }
    for (int e = a0; e < m; ++e) {
      const int k = T.inc[e];
      acc += -(s.P[k] * gQ[k]);
    }
    const int nd = n.jnode[p];
    const int es = s.eslot[p];
    s.V0[p] = (acc - (es >= 0 ? s.em_emh[es] : 0.0) * gE[nd]) - gH[nd];
  }
  bool any_act = false;
  for (int i = gtid<NT>(); i < n.npcv; i += NT) any_act |= s.S[n.pcv_link[i]] == WDS_ACTIVE;
  any_act = gsync_or<NT>(any_act);
  double* lam = s.V1;
  double* t = s.V2;
  if (!any_act) {
    solve_refined<NT, FT>(n, T, s, s.V0, -1, lam, t, 2);
  } else {
    const int p = n.npcv;
    double* scr = w.scr + (size_t)slot * w.nscr * n.Nj;
    double* r2 = scr;
    double* res = r2 + n.Nj;
    double* sx = res + n.Nj;
    double* cols = sx + n.Nj;                 // p Woodbury columns
    double* C = s.small;
    double* y = C + p * p;
    double* actf = y + p;
    if (gtid<NT>() == 0)
      for (int i = 0; i < p; ++i) actf[i] = s.S[n.pcv_link[i]] == WDS_ACTIVE ? 1.0 : 0.0;
    for (int q = gtid<NT>(); q < n.Nj; q += NT) r2[q] = s.V0[q];
    gsync<NT>();
    if (gtid<NT>() == 0)
      for (int i = 0; i < p; ++i)
        // row jc: lam[n2] - lam[n1] = gQ of the free valve flow, i.e.
        // lam[jc] - lam[jo] = sgn gQ (PRV jc = n2, PSV jc = n1)
        if (actf[i] != 0.0) r2[n.pcv_jc[i]] = unit ? 0.0 : n.pcv_sgn[i] * gQ[n.pcv_link[i]];
    gsync<NT>();
    // unrefined solves: the two outer refinement steps below contract their error
    solve_refined<NT, FT>(n, T, s, r2, -1, lam, t, 0);
    for (int c = 0; c < p; ++c) {
      if (actf[c] == 0.0) {  // meets y = 0 in the correction
        for (int q = gtid<NT>(); q < n.Nj; q += NT) cols[(size_t)c * n.Nj + q] = 0.0;
        gsync<NT>();
        continue;
      }
      solve_refined<NT, FT>(n, T, s, nullptr, n.pcv_jc[c], cols + (size_t)c * n.Nj, t, 0);
    }
    if (gtid<NT>() == 0)
      for (int a0 = 0; a0 < p; ++a0)
        for (int c = 0; c < p; ++c) {
          const double cw = cols[(size_t)c * n.Nj + n.pcv_jc[a0]] - cols[(size_t)c * n.Nj + n.pcv_jo[a0]];
          C[a0 * p + c] = cw * actf[a0] * actf[c] + (a0 == c ? 1.0 - actf[a0] : 0.0);
        }
    gsync<NT>();
    auto wood = [&](double* x, const double* rr) {
      if (gtid<NT>() == 0) {
        double* Cc = actf + p;  // working copy, p^2 after C, y, actf in the small buffer
        for (int i = 0; i < p * p; ++i) Cc[i] = C[i];
        for (int a0 = 0; a0 < p; ++a0)
          y[a0] = (x[n.pcv_jc[a0]] - x[n.pcv_jo[a0]] - rr[n.pcv_jc[a0]]) * actf[a0];
        dense_solve(Cc, y, p);
      }
      gsync<NT>();
      for (int q = gtid<NT>(); q < n.Nj; q += NT) {
        double acc = 0.0;
        for (int c = 0; c < p; ++c) acc += cols[(size_t)c * n.Nj + q] * y[c];
        x[q] = x[q] - acc;
      }
      gsync<NT>();
    };
    wood(lam, r2);
    for (int it = 0; it < 2; ++it) {
      for (int q = gtid<NT>(); q < n.Nj; q += NT) res[q] = r2[q] - amul_node(n, T, s, q, lam);
      gsync<NT>();
      if (gtid<NT>() == 0)
        for (int i = 0; i < p; ++i)
          if (actf[i] != 0.0)
            res[n.pcv_jc[i]] = r2[n.pcv_jc[i]] - (lam[n.pcv_jc[i]] - lam[n.pcv_jo[i]]);
      gsync<NT>();
      solve_refined<NT, FT>(n, T, s, res, -1, sx, t, 0);
      wood(sx, res);
      for (int q = gtid<NT>(); q < n.Nj; q += NT) lam[q] = lam[q] + sx[q];
      gsync<NT>();
    }
  }
  // theta contraction
  if (unit) {
    const double* dr = w.dr + (size_t)bf * n.L;
    double* gr = a.gr + (size_t)b * n.L;
    for (int k = gtid<NT>(); k < n.L; k += NT) {
      const double l1 = junc_of(T.e1[k], lam), l2 = junc_of(T.e2[k], lam);
      gr[k] = s.P[k] * (l2 - l1) * dr[k];
    }
    return;
  }
  double* gd = a.gd + (size_t)b * n.N;
  double* gke = a.gke + (size_t)b * n.N;
  double* grh = a.grh + (size_t)b * n.N;
  double* gr = a.gr + (size_t)b * n.L;
  const double* hge = w.hge + (size_t)bf * n.Nj;
  const double* dke = w.dke + (size_t)bf * n.Nj;
  for (int p = gtid<NT>(); p < n.Nj; p += NT) {
    const int nd = n.jnode[p];
    gd[nd] = lam[p];
    double g = 0.0;
    if (s.eslot[p] >= 0) {
      const double lam_e = (gE[nd] + lam[p]) / hge[p];
      g = -(lam_e * dke[p]);
    }
    gke[nd] = g;
    grh[nd] = 0.0;
  }
  const double* dr = w.dr + (size_t)bf * n.L;
  for (int k = gtid<NT>(); k < n.L; k += NT) {
    const double l1 = junc_of(T.e1[k], lam), l2 = junc_of(T.e2[k], lam);
    const double lam_l = s.P[k] * (gQ[k] - (l2 - l1));
    gr[k] = -(lam_l * dr[k]);
    if (a.gsp) {  // pump theta (dgga/autodiff.py:736-741): -lam_l d hloss / d theta
      const int ip = n.link_pump[k];
      double g0 = 0.0, g1 = 0.0, g2 = 0.0;
      if (ip >= 0) {
        const double* dp = w.dpump + (size_t)bf * 3 * n.npump;
        g0 = -(lam_l * dp[ip]);
        g1 = -(lam_l * dp[n.npump + ip]);
        g2 = -(lam_l * dp[2 * n.npump + ip]);
      }
      a.gsp[(size_t)b * n.L + k] = g0;
      a.gh0[(size_t)b * n.L + k] = g1;
      a.grp[(size_t)b * n.L + k] = g2;
    }
  }
  for (int f = gtid<NT>(); f < n.Nf; f += NT) {
    const int nd = n.fnode[f];
    double acc = 0.0;
    for (int e = n.finc_ptr[f]; e < n.finc_split[f]; ++e) {
      const int k = n.finc[e];
      const double l1 = junc_of(T.e1[k], lam), l2 = junc_of(T.e2[k], lam);
      acc += s.P[k] * (gQ[k] - (l2 - l1));
    }
    for (int e = n.finc_split[f]; e < n.finc_ptr[f + 1]; ++e) {
      const int k = n.finc[e];
      const double l1 = junc_of(T.e1[k], lam), l2 = junc_of(T.e2[k], lam);
      acc += -(s.P[k] * (gQ[k] - (l2 - l1)));
    }
    grh[nd] = acc + gH[nd];
    gd[nd] = 0.0;
    gke[nd] = 0.0;
  }
}

template <int NT, class TB, class FT>
__device__ __forceinline__ void adjoint_body(const DevNet& n, const DevWork& w, const AdjArgs& a,
                                             int state_bytes, int blk, int nblk, int groups) {
  const int slot = blk * groups + (int)(threadIdx.x / NT);
  cta_rounds<NT, TB>(n, w, a.B, state_bytes, blk, nblk, groups, [&](const TB& T, Sh s, int b) {
    adjoint_one<NT, TB, FT>(n, w, a, T, s, b, a.by_slot ? slot : b);
  }, a.by_slot != 0);
}

// ---------------------------------------------------------------- unrolled-K reverse
// dP/dq, dY/dq, dP/dr, dY/dr of one link on the branch its coefficients took
// (the formulas of solve_unrolled, dgga/autodiff.py:1495-1591, differentiated
// as autograd does: a clamped quantity is a constant, |q| is q sgn with sgn
// constant; a custom pump curve's segment is chosen from the detached flow).
__device__ void link_dcoef(const DevNet& n, int k, double q, int st, double r, double& Pq,
                           double& Yq, double& Pr, double& Yr) {
  Pq = Yq = Pr = Yr = 0.0;
  const int kd = n.kind[k];
  if (st <= WDS_CLOSED || (n.flags[k] & WDS_F_ZERO_SPEED)) {  // P = 1/CBIG, Y = q
    Yq = 1.0;
    return;
  }
  const double sgn = q < 0.0 ? -1.0 : 1.0, qa = q * sgn;
  double hg, hl, dhg, dhl;
  if (kd <= WDS_KIND_CVPIPE) {
    const double ex = n.hexp, qc = fmax(qa, 1e-30);
    const double pw = pow_pos(qc, ex - 1.0), hg0 = ex * r * pw, rex = n.rhexp;
    const bool lin = hg0 < n.rqtol;
    hg = lin ? n.rqtol : hg0;
    hl = lin ? hg * qa : quotient(hg * qa, ex, rex);
    dhg = (lin || !(qa > 1e-30)) ? 0.0 : ex * (ex - 1.0) * r * (pw / qc);
    dhl = lin ? n.rqtol : quotient(dhg * qa, ex, rex) + quotient(hg, ex, rex);
    const double dhg_r = lin ? 0.0 : ex * pw;
    const double dhl_r = quotient(dhg_r * qa, ex, rex);
    const double km = n.km[k];
    if (km > 0.0) {
      hl += km * qa * qa;
      dhl += 2.0 * km * qa;
      hg += 2.0 * km * qa;
      dhg += 2.0 * km;
    }
    const double h2 = hg * hg, rh2 = recip(h2);
    Pq = quotient(-dhg * sgn, h2, rh2);
    Yq = quotient(dhl * hg - hl * dhg, h2, rh2);
    Pr = quotient(-dhg_r, h2, rh2);
    Yr = quotient(sgn * (dhl_r * hg - hl * dhg_r), h2, rh2);
    return;
  }
  if (kd == WDS_KIND_TCV) {
    const double km = n.km_tcv[k];
    if (!(km > 0.0)) {
      Yq = 1.0;
      return;
    }
    const double hg0 = 2.0 * km * qa;
    const bool lin = hg0 < n.rqtol;
    hg = lin ? n.rqtol : hg0;
    dhg = lin ? 0.0 : 2.0 * km * sgn;
    hl = lin ? q * hg : q * hg / 2.0;
    dhl = lin ? hg : (hg + q * dhg) / 2.0;
    Pq = -dhg / (hg * hg);
    Yq = (dhl * hg - hl * dhg) / (hg * hg);
    return;
  }
  if (kd != WDS_KIND_PUMP) return;
  const int t = n.ptype[k];
  if (t == 3) {  // NOCURVE: P const, Y = q
    Yq = 1.0;
    return;
  }
  const double spc = fmax(n.pspeed[k], 1e-12);
  if (t == 2) {  // CUSTOM, segment frozen: hg const, hl = H0 w^2 + hg q
    Yq = 1.0;
    return;
  }
  const double pn = n.pn[k];
  const double h0e = spc * spc * n.ph0[k];
  const double re = n.pr[k] * pow_pos(spc, 2.0 - pn);
  if (t == 0) {  // CONST_HP
    const double qa2 = fmax(qa * qa, 1e-30);
    const double raw = -re / qa2;
    const bool big = raw > kCBIG, sml = raw < n.rqtol;
    hg = big ? kCBIG : (sml ? n.rqtol : raw);
    dhg = (big || sml || !(qa * qa >= 1e-30)) ? 0.0 : 2.0 * re / (qa2 * qa2) * qa * sgn;
    const double qcc = sgn * fmax(qa, 1e-30);
    hl = (big || sml) ? -hg * q : re / qcc;
    dhl = (big || sml) ? -hg : (qa > 1e-30 ? -re / (qcc * qcc) : 0.0);
  } else if (pn == 1.0) {  // linear
    hg = re;
    dhg = 0.0;
    hl = h0e + re * q;
    dhl = re;
  } else {  // power function
    const double qc = fmax(qa, 1e-30);
    const double raw = pn * re * pow_pos(qc, pn - 1.0);
    const bool sml = raw < n.rqtol;
    hg = sml ? n.rqtol : raw;
    dhg = (sml || !(qa > 1e-30)) ? 0.0 : pn * (pn - 1.0) * re * pow_pos(qc, pn - 2.0) * sgn;
    const double nn = fmax(pn, 1e-30);
    hl = sml ? h0e + hg * q : h0e + hg * q / nn;
    dhl = sml ? hg : (dhg * q + hg) / nn;
  }
  Pq = -dhg / (hg * hg);
  Yq = (dhl * hg - hl * dhg) / (hg * hg);
}

// Derivatives of an emitter's hloss and hgrad in its flow e and its Ke.
__device__ __forceinline__ void emitter_dcoef(const DevNet& n, double e, double ke, double hge,
                                              double& hle_e, double& hge_e, double& hle_k,
                                              double& hge_k) {
  const double kea = fmax(ke, kCSMALL), dkea = ke > kCSMALL ? 1.0 : 0.0;
  const double ae = fabs(e), ea = fmax(ae, 1e-30);
  const double sg = e > 0.0 ? 1.0 : (e < 0.0 ? -1.0 : 0.0);
  const bool lin = n.qexp * kea * pow_pos(ea, n.qexp - 1.0) < n.rqtol;
  hge_e = (lin || !(ae > 1e-30)) ? 0.0 : n.qexp * (n.qexp - 1.0) * kea * pow_pos(ea, n.qexp - 2.0) * sg;
  hge_k = lin ? 0.0 : n.qexp * pow_pos(ea, n.qexp - 1.0) * dkea;
  hle_e = lin ? n.rqtol : (hge_e * e + hge) / n.qexp;
  hle_k = lin ? 0.0 : hge_k * e / n.qexp;
}

// Reverse pass of the unrolled-K map (solve_unrolled's autograd,
// dgga/autodiff.py:1357-1664) for one scenario group.  From the record of the
// forward, iteration k's coefficients, node matrix and factor are rebuilt
// (the same functions as the forward), then:
//   q' = q - (Y - P dh): qb -> Yb, Pb, dh_b (or qb / 2 on the constant-HP half step)
//   e' = e - (hle - (H - el)) / hge: eb -> hle_b, hge_b, H_b
//   H = A^{-1} F:       Fb = A^{-1} H_b (A symmetric), Pb -= (Fb1 - Fb2)(H1 - H2)
//   F = Y terms + P H_fixed + emitter terms + Xflow(q, e, d)
// and the coefficients' derivatives carry Pb, Yb, hle_b, hge_b to the flows,
// emitter flows, resistances and Ke.  Node sums gather over the incidence
// lists (no atomics).  Scratch per scenario: qb [L], a link temporary [L],
// eb [Nj], Fb [Nj].
template <int NT, class TB, class FT>
__device__ __forceinline__ void unrolled_one(const DevNet& n, const DevWork& w, const UnrollArgs& u,
                                             const TB& T, Sh s, int b) {
  const int tid = gtid<NT>();
  s.q = w.lk + (size_t)b * 2 * n.L;
  s.Y = s.q + n.L;
  if (!n.msm) s.Mg = w.M + (size_t)b * n.nT * top_ld(n.nT);
  const double* rrow = u.r + (long long)b * u.r_stride;
  const double* kerow = u.ke + (long long)b * u.ke_stride;
  const double* drow = u.d + (size_t)b * n.N;
  const double* rhrow = u.rh + (size_t)b * n.N;
  FwdArgs a0{};  // the network's own pump parameters
  const PumpTh th = pump_th(n, a0, b);
  double* dj = w.dj + (size_t)b * n.Nj;  // junction demands in elimination order
  for (int p = tid; p < n.Nj; p += NT) dj[p] = drow[n.jnode[p]];
  for (int f = tid; f < n.Nf; f += NT) s.hf[f] = rhrow[n.fnode[f]];
  for (int k = tid; k < n.L; k += NT) s.S[k] = u.s0 ? u.s0[(size_t)b * n.L + k] : n.status0[k];
  gsync<NT>();
  if (!build_emitters<NT>(n, s, kerow, 1)) return;  // uniform; the forward failed alike
  double* qb = u.scr + (size_t)b * (2 * n.L + 2 * n.Nj);
  double* tl = qb + n.L;
  double* eb = tl + n.L;
  double* Fb = eb + n.Nj;
  double* gd = u.gd + (size_t)b * n.N;
  double* grh = u.grh + (size_t)b * n.N;
  double* gke = u.gke + (size_t)b * n.N;
  double* gr = u.gr + (size_t)b * n.L;
  const double* gH = u.gH + (size_t)b * n.N;
  for (int i = tid; i < n.N; i += NT) {
    gd[i] = 0.0;
    grh[i] = 0.0;
    gke[i] = 0.0;
  }
  for (int k = tid; k < n.L; k += NT) {
    gr[k] = 0.0;
    qb[k] = u.gQ[(size_t)b * n.L + k];
  }
  for (int p = tid; p < n.Nj; p += NT)
    eb[p] = s.eslot[p] >= 0 ? u.gE[(size_t)b * n.N + n.jnode[p]] : 0.0;
  gsync<NT>();
  const int R = n.L + 2 * n.Nj;
  const double* recb = u.rec + (size_t)b * u.K * R;
  for (int kk = u.K - 1; kk >= 0; --kk) {
    const double* rr = recb + (size_t)kk * R;
    const bool last = kk == u.K - 1;
    for (int k = tid; k < n.L; k += NT) s.q[k] = rr[k];
    for (int p = tid; p < n.Nj; p += NT) {
      const int es = s.eslot[p];
      if (es >= 0) s.em_e[es] = rr[n.L + p];
    }
    gsync<NT>();
    link_pass<NT>(n, th, T, s, rrow, w.hge + (size_t)b * n.Nj);
    gsync<NT>();
    assemble_gga<NT, FT>(n, T, s, dj, w.hge + (size_t)b * n.Nj);
    factor<NT, FT>(n, T, s);  // the forward factored this matrix: positive definite
    for (int p = tid; p < n.Nj; p += NT) s.V1[p] = rr[n.L + n.Nj + p];
    gsync<NT>();
    // (1) q' = q - dq: the head-difference adjoint of each link
    for (int k = tid; k < n.L; k += NT) {
      const double dh = head_of(T.e1[k], s.V1, s.hf) - head_of(T.e2[k], s.V1, s.hf);
      const double dq = s.Y[k] - s.P[k] * dh;
      const bool hit = (n.flags[k] & WDS_F_CHP) && dq > s.q[k];
      tl[k] = hit ? 0.0 : qb[k] * s.P[k];
    }
    gsync<NT>();
    // (2) H_b at the junctions (links, emitter update, output) -> V0; fixed heads -> grh
    for (int p = tid; p < n.Nj; p += NT) {
      double acc = 0.0;
      const int a = T.inc_ptr[p], m = T.inc_split[p], z = T.inc_ptr[p + 1];
      for (int e = a; e < m; ++e) acc += tl[T.inc[e]];
      for (int e = m; e < z; ++e) acc += -tl[T.inc[e]];
      if (last) acc += gH[n.jnode[p]];
      const int es = s.eslot[p];
      if (es >= 0) {
        double hle, hge;
        emitter_hl(n, s.em_e[es], s.em_ke[es], hle, hge);
        acc += eb[p] / hge;  // e' = e - (hle - (H - el)) / hge: de'/dH = 1/hge
      }
      s.V0[p] = acc;
    }
    for (int f = tid; f < n.Nf; f += NT) {
      double acc = 0.0;
      for (int e = n.finc_ptr[f]; e < n.finc_split[f]; ++e) acc += tl[n.finc[e]];
      for (int e = n.finc_split[f]; e < n.finc_ptr[f + 1]; ++e) acc += -tl[n.finc[e]];
      if (last) acc += gH[n.fnode[f]];
      grh[n.fnode[f]] += acc;
    }
    gsync<NT>();
    // (3) F_b = A^{-1} H_b
    solve_refined<NT, FT>(n, T, s, s.V0, -1, Fb, s.V2, 2);
    // (4) links: P_b, Y_b from q', A and F; carried to q and r
    for (int k = tid; k < n.L; k += NT) {
      const double q = s.q[k], P = s.P[k], Y = s.Y[k];
      const int c1 = T.e1[k], c2 = T.e2[k];
      const double dh = head_of(c1, s.V1, s.hf) - head_of(c2, s.V1, s.hf);
      const bool hit = (n.flags[k] & WDS_F_CHP) && (Y - P * dh) > q;
      const double dqb = -qb[k];
      const double uu = junc_of(c1, Fb) - junc_of(c2, Fb);
      const double vv = junc_of(c1, s.V1) - junc_of(c2, s.V1);
      double Pb = (hit ? 0.0 : -dqb * dh) - uu * vv;
      const double Yb = (hit ? 0.0 : dqb) + uu;
      double tg = 0.0;  // F = ... + P H_fixed at the junction end
      if (c1 < 0 && c2 >= 0) {
        Pb += Fb[c2] * s.hf[-c1 - 1];
        tg = Fb[c2] * P;
      } else if (c2 < 0 && c1 >= 0) {
        Pb += Fb[c1] * s.hf[-c2 - 1];
        tg = Fb[c1] * P;
      }
      tl[k] = tg;
      double Pq, Yq, Pr, Yr;
      link_dcoef(n, k, q, s.S[k], rrow[k], Pq, Yq, Pr, Yr);
      qb[k] = qb[k] + (hit ? dqb / 2.0 : 0.0) - uu + Pb * Pq + Yb * Yq;
      gr[k] += Pb * Pr + Yb * Yr;
    }
    gsync<NT>();
    // (5) fixed heads through the grounding terms; junctions: demand, emitters
    for (int f = tid; f < n.Nf; f += NT) {
      double acc = 0.0;
      for (int e = n.finc_ptr[f]; e < n.finc_ptr[f + 1]; ++e) acc += tl[n.finc[e]];
      grh[n.fnode[f]] += acc;
    }
    for (int p = tid; p < n.Nj; p += NT) {
      const double Fp = Fb[p];
      gd[n.jnode[p]] += -Fp;
      const int es = s.eslot[p];
      if (es < 0) continue;
      const double ee = s.em_e[es], ke = s.em_ke[es];
      double hle, hge, hle_e, hge_e, hle_k, hge_k;
      emitter_hl(n, ee, ke, hle, hge);
      emitter_dcoef(n, ee, ke, hge, hle_e, hge_e, hle_k, hge_k);
      const double dqe = (hle - (s.V1[p] - n.el[p])) / hge;
      const double dqeb = -eb[p];
      const double hleb = dqeb / hge + Fp / hge;
      const double hgeb = -dqeb * dqe / hge + Fp * s.V1[p] / (hge * hge) -
                          Fp * (hle + n.el[p]) / (hge * hge);
      eb[p] = eb[p] - Fp + hleb * hle_e + hgeb * hge_e;
      gke[n.jnode[p]] += hleb * hle_k + hgeb * hge_k;
    }
    gsync<NT>();
  }
}

template <int NT, class TB, class FT>
__device__ __forceinline__ void unrolled_body(const DevNet& n, const DevWork& w, const UnrollArgs& u,
                                              int state_bytes, int blk, int nblk, int groups) {
  cta_rounds<NT, TB>(n, w, u.B, state_bytes, blk, nblk, groups, [&](const TB& T, Sh s, int b) {
    unrolled_one<NT, TB, FT>(n, w, u, T, s, b);
  });
}

template <int NT, int GR, class TB, class FT>
__global__ void __launch_bounds__(NT * GR, 1) k_unrolled(DevNet n, DevWork w, UnrollArgs u,
                                                         int state_bytes) {
  unrolled_body<NT, TB, FT>(n, w, u, state_bytes, blockIdx.x, gridDim.x, GR);
}

template <int NT, int GR, class TB, class FT>
__global__ void __launch_bounds__(NT * GR, 1) k_forward(DevNet n, DevWork w, FwdArgs a,
                                                        int state_bytes) {
  forward_body<NT, TB, FT>(n, w, a, state_bytes, blockIdx.x, gridDim.x, GR);
}

template <int NT, int GR, class TB, class FT>
__global__ void __launch_bounds__(NT * GR, 1) k_adjoint(DevNet n, DevWork w, AdjArgs a,
                                                        int state_bytes) {
  adjoint_body<NT, TB, FT>(n, w, a, state_bytes, blockIdx.x, gridDim.x, GR);
}

// Several plans (networks of different sizes) in one launch of 1024-thread
// CTAs: CTAs [job.cta0, next job's cta0) run the job's plan, a small network
// with J.groups groups of 256 threads (the others idle), a large one with one
// scenario per CTA.
template <class FT>
__global__ void __launch_bounds__(kWideThreads, 1)
    k_forward_multi(const __grid_constant__ FwdJobs jobs) {
  int p = 0;
  while (p + 1 < jobs.n && (int)blockIdx.x >= jobs.j[p + 1].cta0) ++p;
  const FwdJob& J = jobs.j[p];
  const int ctas = (J.a.B + J.groups - 1) / J.groups, c = blockIdx.x - J.cta0;
  if (J.n.wide)
    forward_body<kWideThreads, LTab, FT>(J.n, J.w, J.a, J.state_bytes, c, ctas, 1);
  else
    forward_body<256, STab, FT>(J.n, J.w, J.a, J.state_bytes, c, ctas, J.groups);
}

template <class FT>
__global__ void __launch_bounds__(kWideThreads, 1)
    k_adjoint_multi(const __grid_constant__ AdjJobs jobs) {
  int p = 0;
  while (p + 1 < jobs.n && (int)blockIdx.x >= jobs.j[p + 1].cta0) ++p;
  const AdjJob& J = jobs.j[p];
  const int ctas = (J.a.B + J.groups - 1) / J.groups, c = blockIdx.x - J.cta0;
  if (J.n.wide)
    adjoint_body<kWideThreads, LTab, FT>(J.n, J.w, J.a, J.state_bytes, c, ctas, 1);
  else
    adjoint_body<256, STab, FT>(J.n, J.w, J.a, J.state_bytes, c, ctas, J.groups);
}

}  // namespace

// Kernel selectors, one definition per instance source and factor precision
// (declared in wds_internal.h): the host stub of the kernel for the plan's
// layout and scenario groups per CTA.
#ifndef WDS_FP32
#define WDS_FP32 0
#endif
#if WDS_FP32
using KFT = float;
#define WDS_KSEL(name) name##_f32
#else
using KFT = double;
#define WDS_KSEL(name) name##_f64
#endif

}  // namespace wds
