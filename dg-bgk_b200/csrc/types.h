// Data layout shared by the host plan builder and the sm_100a kernels.
//
// HBM layout of the distribution function: f[(e*3 + i)*Vp + v] -- element e
// (in the plan's locality order), DG node i (0..2), discrete velocity v
// fastest, rows padded to a pitch Vp (a multiple of 32 velocities, so every
// row starts on a 128-byte boundary and splits into whole 128-byte sweep
// segments).  The padding velocities hold zeros forever (the buffers are
// cleared at allocation and the kernels write zeros there), so kernels may
// read whole 16-byte vectors past V without bounds checks.  Two such buffers are
// kept (ping-pong): within one pseudo-time step the reference updates every
// element of velocity IV only after all edge fluxes of IV are formed
// (src/advnce.f90:321-367), i.e. a Jacobi update in space, so the sweep reads
// f^n and writes f^{n+1}.
#pragma once
#include <cstdint>

#include "exp_tang.h"

namespace dgbgk {

// A row of a sweep tile in bytes: one velocity segment of a DG node.  The
// first row of a tile holds zeros, row r = 3*slot + i comes after it.
constexpr int ROW_BYTES = 128;
constexpr unsigned tile_row(int r) { return (unsigned)(r + 1) * ROW_BYTES; }

// A coefficient of an element record.  FP32: the value twice, the operand of
// a packed instruction on two velocities as it is loaded (duplicating in
// registers took one ALU instruction per coefficient and use); FP64: the
// value.
struct alignas(8) CoefF {
  float x, y;
};
template <class T> struct CoefOf;
template <> struct CoefOf<float> {
  using type = CoefF;
};
template <> struct CoefOf<double> {
  using type = double;
};
#if defined(__CUDACC__)
__host__ __device__
#endif
inline void coef_set(CoefF& c, double v) { c.x = c.y = (float)v; }
#if defined(__CUDACC__)
__host__ __device__
#endif
inline void coef_set(double& c, double v) { c = v; }

// Everything the sweep needs about one element, in one 16-byte-aligned
// record.  The leading part (shape-function gradients and the GTEQNF /
// COMPMU parameters of the three DG nodes, 21 coefficients) is all a halo
// element needs; the moment kernel rewrites the node parameters every step.
//
// Per local edge k (from local node k to node (k+1) mod 3) the sweep forms
// the flux from an upwind "source" row set: the neighbour across an interior
// side, the element itself on an outflow side (the upwind value of an outflow
// side is always the element's own) and the tile's row of zeros on wall
// sides (the wall's own flux is added by a separate path) and on inflow sides
// (no flux; the part the element's own values add is taken out by the same
// path).  The source's two rows (its local nodes at my points k and k+1) are
// given as their byte offsets in the sweep tile (tile_row).
template <class T> struct alignas(16) ElemRec {
  using C = typename CoefOf<T>::type;
  C gx[3], gy[3];  // shape-function gradients GEOME(1:3), GEOME(4:6)
  // GTEQNF's Maxwellian NFO (src/gteqnf.f90:26-40) at node i and velocity c,
  // with A = DISND*BETA2/PI and u = (DISUX, DISUY):
  //  FP32: NFO = A * 2^(ex*|c-u|^2), ex = -BETA2*log2(e): A, ex, and -u in
  //        ux, uy;
  //  FP64: NFO = exp(a0 + a1*cx + a2*cy + ex*|c|^2), the exponent expanded:
  //        A holds a0 = ln(A) - BETA2*|u|^2, ux a1 = 2*BETA2*ux, uy a2 =
  //        2*BETA2*uy, ex = -BETA2 (a0 = -inf where A = 0).
  // (NFO = 0 where DISPS < 1e-20, src/gteqnf.f90:32.)
  C A[3];
  C ex[3];
  C ux[3];
  C uy[3];
  C mu[3];     // collision frequency MU (src/compmu.f90:90-92)
  C pad;
  C mt[3];     // MU again, for the update of the element's own values
  C mm[3];     // MMAT (IMMAT = 1) or CMMAT row sums (IMMAT = 0)
  C en[3][2];  // per edge -AL times the outward unit normal, AL = EL/6 (interior) or RSIDO(3)/6 (boundary)
  unsigned off[3][2];  // per edge: tile offsets of the source's rows at points k and k+1
  int bside[3];  // boundary side index of each wall edge (kind 3), else -1
  int flags;  // bits [0,3): DG node i sits on an inflow-side node (INFLOW);
              // bits [3,6): edge k is a wall side; bits [6,9): edge k is an
              // inflow side
  int wslot;  // wall element slot (ALPHA < 1: the deferred updates), else -1
};
constexpr int FLAG_INFLOW_EDGE0 = 1 << 6;  // FLAG_INFLOW_EDGE0 << k: edge k is an inflow side
static_assert(sizeof(ElemRec<float>) == 320 && sizeof(ElemRec<double>) == 320, "record layout");
// coefficients of the leading part a halo element needs (gx .. mu)
constexpr int REC_HEAD_VALUES = 21;

// One type-4 wall side for the wall-flux kernel (FLUCON2).
struct WallSide {
  int elem;     // plan order
  int in1, in2; // local nodes of BSIDO(1), BSIDO(2) in that element
  int bside;    // boundary side index
  double anx, any;     // RSIDO(1:2)
  double sumbottom;    // sqrt(2*PI*R^3*T_w^3)
};

// One type-4 wall side for GETFOR's lift and drag (src/getfor.f90:29-49):
// its two nodes and LEN*PERP, PERP the unit normal of the side vector
// turned 90 degrees anticlockwise.
struct ForceSide {
  int ip1, ip2;  // nodes BSIDO(1), BSIDO(2), 0-based
  double lx, ly; // LEN*PERP(1), LEN*PERP(2)
};

// Device-side control block of one case.
struct Ctrl {
  int done;       // kernels skip the case when set
  int step;       // steps run in this advance call
  int max_steps;
  int nonfinite;  // set when a residual was NaN/Inf
  double tol;     // relative L2 tolerance (<= 0: none)
  double ref;     // reference L2 residual (0: take the first step's)
  double maxmu;   // max MU of the current step (atomicMax on the bits; reset by resid_book)
  double dtc;     // Courant limit DTEc (src/alotim.f90)
  double acc_sq;  // sum of squared changes of the current step (sweep atomics; reset by resid_book)
  double acc_max; // max residual of the current step (atomicMax on the bits; reset by resid_book)
  int cur;        // which f buffer holds the current state (resid_book swaps it)
  int timeout;    // set when a bounded device wait gave up
  int itime0;     // steps the handle ran before this advance call (the reference's ITIME - step - 1)
  int pad0;
};

// Device-side control of one launch set (a case alone or a batch).
struct BatchCtl {
  int sweep_next;  // sweep work units handed out beyond the first wave
  int sweep_done;  // sweep CTAs that have finished (both reset by the last one)
  int pad[14];
  double etab[EXP_TAB];  // 2^(j/256) of the FP64 sweep's exp
};

}  // namespace dgbgk
