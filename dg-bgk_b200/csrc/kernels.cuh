// sm_100a kernels of the DG-BGK pseudo-time step.
//
// One step (src/advnce.f90:220-400) is three launches (with ALPHA < 1 also
// k_wspec and k_resid after the sweep):
//   k_moments : MACROS passes 1+2 (src/macros.f90:80-154) fused with COMPMU
//               (src/compmu.f90:36-97) and the GTEQNF parameters
//               (src/gteqnf.f90:26-40).  Persistent warps take R whole
//               velocity rows of f at a time (32/R lanes per row) from a
//               per-warp ring of stages filled by 1-D bulk copies, so f is
//               read from HBM once for both passes; every access is a
//               16-byte vector.
//   k_wall    : FLUCON2 (src/flucon2.f90:134-233), one CTA per wall side.
//   k_sweep   : the whole velocity-loop body (GTEQNF, GETFLA, GETELC,
//               EDGFLXOPT/GETBOU, GETINC/CMMINC, ADTHEM, INFLOW;
//               src/advnce.f90:286-377) on tiles of (element block x one
//               128-byte velocity segment).  Persistent CTAs draw work units
//               (a block at several tiles); the block's records are staged
//               once per unit, the tiles' f rows arrive by cp.async,
//               double-buffered, and eight lanes share an element, each at 4
//               (FP32, packed pairs) or 2 (FP64) velocities.
//               Its last CTA does GETRES + the residual bookkeeping
//               (src/advnce.f90:385, 422-429), the convergence test and the
//               step counter.
// Every device-side wait on an mbarrier is bounded: on expiry the kernel
// sets Ctrl::timeout, drains its own copies with a second bounded wait and
// returns; the host reports DGBGK_ECUDA.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "exp_tang.h"
#include "pdl.cuh"
#include "types.h"

namespace dgbgk {

constexpr double PI_D = 3.1416;  // the reference's PI
constexpr double TINY_D = 1e-20;
constexpr double LOG2E_D = 1.4426950408889634;  // log2(e)
constexpr unsigned WAIT_TRIES = 1u << 22;  // x ~256 ns sleep: ~1 s

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------- TMA / mbarrier helpers ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase with the given parity.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  for (unsigned i = 0; i < WAIT_TRIES; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i > 32) __nanosleep(256);
  }
  return false;
}
// 1-D bulk copy global -> shared (16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// -------------------------------------------------------------- cases ----
// One case (a mesh, its velocity grid and its state) as the kernels see it.
// Every launch works on a table of cases: a single handle is a table of one,
// a batch a table of many.  The work of the launch set is flattened: sweep
// units, moment row groups and wall sides of case c are [off[c], off[c+1]).
template <class T> struct alignas(64) CaseDev {
  T* f[2];            // state, ping-pong; Ctrl::cur is the current one
  ElemRec<T>* rec;
  const int* halo;  // [nblocks][hp]: the block's halo count and its halo elements
  int hp;           // pitch: at least one more than the largest halo
  const T* swtab;  // [NTAB][Vp] sweep tables cx, cy, NFINF (, |c|^2), zero past V
  const T* cx;     // rows 0, 1, 2 of swtab
  const T* cy;
  const T* nfinf;
  const T* tabs;   // [MOM_TABS][Vp] moment tables: cx, cy, w = WEIGHT*JAC*FRAC, w*cx, w*cy; zero past V
  T* bwall;        // per boundary side [4]: wall velocity (x, y), the wall Maxwellian's exponent coefficient
                   // -1/(2 R T_w) (FP32: times log2(e)), ALPHA*ETA (written by the wall kernel)
  double* bEtaD;
  const double* cxD;  // [V] FP64 velocity tables for FLUCON2
  const double* cyD;
  const double* wjf;
  const WallSide* walls;
  const T* cmax;   // IMMAT = 0 residual tables
  const T* cmin;
  double* nraw;    // per DG node: INT (number density before the 1e-20 test)
  double* disux;
  double* disuy;
  double* disps;
  double* mu;
  double* hist;  // [step][3] of an advance call: max residual, L2 residual, DTE
  Ctrl* ctrl;
  double MM, sigt;  // M/NA, PI*d*d
  T alpha;
  int E, V, Vp, nblocks, nvt;
  int tpu, nreg, ngrp, halve;  // velocity-tile groups of the sweep's units (sweep_group)
  int nwall;          // FLUCON2 wall sides
  unsigned rowbytes;  // V*sizeof(T) rounded up to 16
  // ALPHA < 1: the specular part of the wall flux (the host plan's tables)
  int spec;                 // 0: ALPHA = 1 or no wall side
  int immat;                // 1: lumped mass (GETINC), 0: CMMINC
  int n_spec_par, n_spec_slots;
  const int* rside;         // [B] reflection-table row, -1 off the walls
  const int* rf_i;          // [rows][V][2] mirrored grid velocities I1, I2; -1 where TEST >= 0
  const T* rf_z;            // [rows][V][2] ZD1, ZD2
  const unsigned* rf_bits;  // [B][rf_words] bit v: rf_i >= 0 there
  int rf_words;             // Vp/32
  const int* welem;         // [slots] wall elements (plan order)
  T* wd;                    // deferred values: IMMAT = 1 [slots][3][Vp] DELUN without the specular part;
                            // IMMAT = 0 [2][slots][3][Vp] RHS*DTE without it, COLL*DTE
  const int* spec_par;      // items slot*V + v
  const int* spec_seq_off;  // [slots + 1]
  const int* spec_seq;      // [items][2]: the item, the end of its level
};

// Size of the next group of the sweep's tail when r tiles remain: half of
// them, rounded up (two or one at the end).
__host__ __device__ inline int sweep_tail_tiles(int r) { return r <= 2 ? r : (r + 1) / 2; }

// Tiles [vt0, vt0 + ntl) of velocity-tile group g: groups below nreg hold
// tpu tiles, the rest is one group or (halve) shrinking groups
// (sweep_tail_tiles).
template <class T> __device__ __forceinline__ void sweep_group(const CaseDev<T>& C, int g, int& vt0, int& ntl) {
  if (g < C.nreg) {
    vt0 = g * C.tpu;
    ntl = C.tpu;
    return;
  }
  int s = C.nreg * C.tpu, r = C.nvt - s;
  if (!C.halve) {
    vt0 = s;
    ntl = r;
    return;
  }
  for (int m = C.nreg; m < g; ++m) {
    const int n = sweep_tail_tiles(r);
    s += n;
    r -= n;
  }
  vt0 = s;
  ntl = sweep_tail_tiles(r);
}

// Moment tables: the row modes read the first three; the element mode of a
// single case (tables in shared memory) rows 2 to 4 in its first pass and 0
// to 2 in its second, of a batch (tables through L1) the first three.
constexpr int MOM_TABS = 5;
template <class T> __host__ __device__ constexpr int mom_tables(int R) { return R == 3 && sizeof(T) == 4 ? 5 : 3; }

template <class T> struct BatchArgs {
  const CaseDev<T>* cases;  // [ncases]
  const int* unit_off;      // [ncases + 1] sweep work units
  const int* grp_off;       // [ncases + 1] moment row groups
  const int* wall_off;      // [ncases + 1] wall sides
  BatchCtl* ctl;
  int ncases;
  int max_halo;             // over the cases (sweep tile layout)
  int sweep_bufs;           // sweep tile buffers, 2 or (a wide halo) 1
  int fuse_resid;           // the sweep's last CTA does the step's bookkeeping (else k_resid)
  int mom_stages;           // moment ring stages per warp
  unsigned mom_rowbytes;    // moment ring row size (max over the cases)
};

// The case c with off[c] <= x < off[c + 1] (cases with empty ranges are
// skipped: the largest c with off[c] <= x).
__device__ __forceinline__ int find_case(const int* __restrict__ off, int n, int x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------ moments ----

// sqrt by a reciprocal-square-root seed and one Newton step for 1/sqrt(x),
// y <- y (3 - x y^2)/2, in FP64 (relative error ~1e-14 from a ~1e-7 seed).
__device__ __forceinline__ float rsqrt_sfu(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ double sqrt_newton(double x) {
  const float xf = (float)x;
  if (!(xf > 0.f)) return 0.0;
  const double y0 = (double)rsqrt_sfu(xf);
  const double t = x * y0;  // sqrt(x) to the seed's accuracy
  return t * fma(-0.5 * y0, t, 1.5);
}
// FP32 sqrt from the SFU (sqrt.approx: relative error ~2^-23; sqrt(0) = 0)
__device__ __forceinline__ float sqrt_fast(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Pass sums over one velocity row in shared memory by the L lanes of a
// group (lane sub takes 16-byte vectors sub, sub+L, ...).  FP64 storage:
// FP64 arithmetic.  FP32 storage: FP32 arithmetic; each lane's partial sums
// (V/(4L) vectors) are converted to FP64 before the group sum.
template <class T> struct RowMath;

template <> struct RowMath<double> {
  static __device__ __forceinline__ void pass1(const double* row, const double* tb, int Vp, int nq, int sub, int L,
                                               double& s0, double& s1, double& s2) {
    const double2* r = reinterpret_cast<const double2*>(row);
    const double2* cx = reinterpret_cast<const double2*>(tb);
    const double2* cy = reinterpret_cast<const double2*>(tb + Vp);
    const double2* wj = reinterpret_cast<const double2*>(tb + 2 * Vp);
    for (int q = sub; q < nq; q += L) {
      const double2 x = r[q], c = cx[q], d = cy[q], w = wj[q];
      const double a0 = w.x * x.x, a1 = w.y * x.y;
      s0 += a0 + a1;
      s1 = fma(c.x, a0, fma(c.y, a1, s1));
      s2 = fma(d.x, a0, fma(d.y, a1, s2));
    }
  }
  static __device__ __forceinline__ void pass2(const double* row, const double* tb, int Vp, int nq, int sub, int L,
                                               double ux, double uy, double& sp, double& sc) {
    const double2* r = reinterpret_cast<const double2*>(row);
    const double2* cx = reinterpret_cast<const double2*>(tb);
    const double2* cy = reinterpret_cast<const double2*>(tb + Vp);
    const double2* wj = reinterpret_cast<const double2*>(tb + 2 * Vp);
    for (int q = sub; q < nq; q += L) {
      const double2 x = r[q], c = cx[q], d = cy[q], w = wj[q];
      const double dx0 = c.x - ux, dy0 = d.x - uy, dx1 = c.y - ux, dy1 = d.y - uy;
      const double q0 = dx0 * dx0 + dy0 * dy0, q1 = dx1 * dx1 + dy1 * dy1;
      const double a0 = w.x * x.x, a1 = w.y * x.y;
      sp = fma(q0, a0, fma(q1, a1, sp));                            // src/macros.f90:144-148, times 2
      sc = fma(sqrt_newton(q0), a0, fma(sqrt_newton(q1), a1, sc));  // src/compmu.f90:71-74
    }
    sp *= 0.5;  // (sp starts at zero)
  }
};

__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

template <> struct RowMath<float> {
  // on packed pairs (fma/add/mul.rn.f32x2): each sum as two partial sums,
  // the halves of one pair (the even and the odd values of a vector)
  static __device__ __forceinline__ void pass1(const float* row, const float* tb, int Vp, int nq, int sub, int L,
                                               double& s0, double& s1, double& s2) {
    const float4* r = reinterpret_cast<const float4*>(row);
    const float4* cx = reinterpret_cast<const float4*>(tb);
    const float4* cy = reinterpret_cast<const float4*>(tb + Vp);
    const float4* wj = reinterpret_cast<const float4*>(tb + 2 * Vp);
    float2 t0 = make_float2(0.f, 0.f), t1 = t0, t2 = t0;
    for (int q = sub; q < nq; q += L) {
      const float4 x = r[q], c = cx[q], d = cy[q], w = wj[q];
      const float2 al = __fmul2_rn(lo2(w), lo2(x)), ah = __fmul2_rn(hi2(w), hi2(x));
      t0 = __fadd2_rn(t0, __fadd2_rn(al, ah));
      t1 = __ffma2_rn(lo2(c), al, __ffma2_rn(hi2(c), ah, t1));
      t2 = __ffma2_rn(lo2(d), al, __ffma2_rn(hi2(d), ah, t2));
    }
    s0 += (double)t0.x + (double)t0.y;
    s1 += (double)t1.x + (double)t1.y;
    s2 += (double)t2.x + (double)t2.y;
  }
  static __device__ __forceinline__ void pass2(const float* row, const float* tb, int Vp, int nq, int sub, int L,
                                               double ux, double uy, double& sp, double& sc) {
    const float2 nx = make_float2(-(float)ux, -(float)ux), ny = make_float2(-(float)uy, -(float)uy);
    const float4* r = reinterpret_cast<const float4*>(row);
    const float4* cx = reinterpret_cast<const float4*>(tb);
    const float4* cy = reinterpret_cast<const float4*>(tb + Vp);
    const float4* wj = reinterpret_cast<const float4*>(tb + 2 * Vp);
    float2 tp = make_float2(0.f, 0.f), tc = tp;
    for (int q = sub; q < nq; q += L) {
      const float4 x = r[q], c = cx[q], d = cy[q], w = wj[q];
      const float2 el = __fadd2_rn(lo2(c), nx), eh = __fadd2_rn(hi2(c), nx);
      const float2 gl = __fadd2_rn(lo2(d), ny), gh = __fadd2_rn(hi2(d), ny);
      const float2 ql = __ffma2_rn(el, el, __fmul2_rn(gl, gl)), qh = __ffma2_rn(eh, eh, __fmul2_rn(gh, gh));
      const float2 al = __fmul2_rn(lo2(w), lo2(x)), ah = __fmul2_rn(hi2(w), hi2(x));
      tp = __ffma2_rn(ql, al, __ffma2_rn(qh, ah, tp));
      const float2 sl = make_float2(sqrt_fast(ql.x), sqrt_fast(ql.y));
      const float2 sh = make_float2(sqrt_fast(qh.x), sqrt_fast(qh.y));
      tc = __ffma2_rn(sl, al, __ffma2_rn(sh, ah, tc));
    }
    sp += 0.5 * ((double)tp.x + (double)tp.y);
    sc += (double)tc.x + (double)tc.y;
  }
};

// Pass sums over the three velocity rows of one element by all 32 lanes of
// a warp (lane l takes 16-byte vectors l, l+32, ...): the velocity tables
// are loaded once per vector for the three rows.  FP32 storage: FP32 lane
// partials, summed in FP64 across the warp; FP64 storage: FP64 throughout.
template <class T> struct ElemMath;

// body(o) for the byte offsets o = 16*q of a lane's vectors, two at a time
// (half the address arithmetic: FP32 0.128 -> 0.124 ms on the 200x100 channel)
template <class F> __device__ __forceinline__ void for_vectors(int lane, int nq, F body) {
  int q = lane;
  for (; q + 32 < nq; q += 64) {
    body(16 * q);
    body(16 * q + 512);
  }
  if (q < nq) body(16 * q);
}
template <class V> __device__ __forceinline__ V at(const unsigned char* p, int o) {
  return *reinterpret_cast<const V*>(p + o);
}

template <> struct ElemMath<float> {
  // Each sum runs as two partial sums, the even and the odd values of a
  // vector (shorter dependent chains: 0.1535 -> 0.1508 ms on the 200x100
  // channel; four partials were slower), the halves of one packed pair
  // (fma/add/mul.rn.f32x2: one instruction for two values; 0.1527 ->
  // 0.1456 ms).
  // pass 1.  TAB: from the tables w, w*cx, w*cy (three FMAs per value;
  // tables in shared memory); otherwise from w, cx, cy (w*f, then three
  // sums; the tables the second pass reads too, through L1)
  template <bool TAB>
  static __device__ __forceinline__ void pass1(const unsigned char* rows, unsigned pitch, const float* tb, int Vp,
                                               int nq, int lane, double (&s)[3][3]) {
    const unsigned char* wj = reinterpret_cast<const unsigned char*>(tb + 2 * Vp);
    const unsigned char* wx = reinterpret_cast<const unsigned char*>(tb + (TAB ? 3 : 0) * Vp);
    const unsigned char* wy = reinterpret_cast<const unsigned char*>(tb + (TAB ? 4 : 1) * Vp);
    float2 t[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) t[r][k] = make_float2(0.f, 0.f);
    for_vectors(lane, nq, [&](int o) {
      const float4 w = at<float4>(wj, o), c = at<float4>(wx, o), d = at<float4>(wy, o);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float4 x = at<float4>(rows + r * pitch, o);
        if constexpr (TAB) {
          t[r][0] = __ffma2_rn(lo2(w), lo2(x), __ffma2_rn(hi2(w), hi2(x), t[r][0]));
          t[r][1] = __ffma2_rn(lo2(c), lo2(x), __ffma2_rn(hi2(c), hi2(x), t[r][1]));
          t[r][2] = __ffma2_rn(lo2(d), lo2(x), __ffma2_rn(hi2(d), hi2(x), t[r][2]));
        } else {
          const float2 al = __fmul2_rn(lo2(w), lo2(x)), ah = __fmul2_rn(hi2(w), hi2(x));
          t[r][0] = __fadd2_rn(t[r][0], __fadd2_rn(al, ah));
          t[r][1] = __ffma2_rn(lo2(c), al, __ffma2_rn(hi2(c), ah, t[r][1]));
          t[r][2] = __ffma2_rn(lo2(d), al, __ffma2_rn(hi2(d), ah, t[r][2]));
        }
      }
    });
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) s[r][k] = (double)t[r][k].x + (double)t[r][k].y;
  }
  // pass 2 on packed pairs (c - u as c + (-u))
  static __device__ __forceinline__ void pass2(const unsigned char* rows, unsigned pitch, const float* tb, int Vp,
                                               int nq, int lane, const float (&u)[3][2], double (&s)[3][2]) {
    const unsigned char* cx = reinterpret_cast<const unsigned char*>(tb);
    const unsigned char* cy = reinterpret_cast<const unsigned char*>(tb + Vp);
    const unsigned char* wj = reinterpret_cast<const unsigned char*>(tb + 2 * Vp);
    float2 nu[3][2], t[3][2];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      nu[r][0] = make_float2(-u[r][0], -u[r][0]);
      nu[r][1] = make_float2(-u[r][1], -u[r][1]);
      t[r][0] = t[r][1] = make_float2(0.f, 0.f);
    }
    for_vectors(lane, nq, [&](int o) {
      const float4 c = at<float4>(cx, o), d = at<float4>(cy, o), w = at<float4>(wj, o);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float4 x = at<float4>(rows + r * pitch, o);
        const float2 el = __fadd2_rn(lo2(c), nu[r][0]), eh = __fadd2_rn(hi2(c), nu[r][0]);
        const float2 gl = __fadd2_rn(lo2(d), nu[r][1]), gh = __fadd2_rn(hi2(d), nu[r][1]);
        const float2 ql = __ffma2_rn(el, el, __fmul2_rn(gl, gl)), qh = __ffma2_rn(eh, eh, __fmul2_rn(gh, gh));
        const float2 al = __fmul2_rn(lo2(w), lo2(x)), ah = __fmul2_rn(hi2(w), hi2(x));
        t[r][0] = __ffma2_rn(ql, al, __ffma2_rn(qh, ah, t[r][0]));  // src/macros.f90:144-148
        const float2 sl = make_float2(sqrt_fast(ql.x), sqrt_fast(ql.y));
        const float2 sh = make_float2(sqrt_fast(qh.x), sqrt_fast(qh.y));
        t[r][1] = __ffma2_rn(sl, al, __ffma2_rn(sh, ah, t[r][1]));  // src/compmu.f90:71-74
      }
    });
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      s[r][0] = 0.5 * ((double)t[r][0].x + (double)t[r][0].y);
      s[r][1] = (double)t[r][1].x + (double)t[r][1].y;
    }
  }
};

template <> struct ElemMath<double> {
  // (from w, cx, cy: the products' tables would take the room of a stage)
  template <bool TAB>
  static __device__ __forceinline__ void pass1(const unsigned char* rows, unsigned pitch, const double* tb, int Vp,
                                               int nq, int lane, double (&s)[3][3]) {
    const unsigned char* cx = reinterpret_cast<const unsigned char*>(tb);
    const unsigned char* cy = reinterpret_cast<const unsigned char*>(tb + Vp);
    const unsigned char* wj = reinterpret_cast<const unsigned char*>(tb + 2 * Vp);
#pragma unroll
    for (int r = 0; r < 3; ++r) s[r][0] = s[r][1] = s[r][2] = 0.0;
    for_vectors(lane, nq, [&](int o) {
      const double2 w = at<double2>(wj, o), c = at<double2>(cx, o), d = at<double2>(cy, o);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double2 x = at<double2>(rows + r * pitch, o);
        const double a0 = w.x * x.x, a1 = w.y * x.y;
        s[r][0] += a0 + a1;
        s[r][1] = fma(c.x, a0, fma(c.y, a1, s[r][1]));
        s[r][2] = fma(d.x, a0, fma(d.y, a1, s[r][2]));
      }
    });
  }
  static __device__ __forceinline__ void pass2(const unsigned char* rows, unsigned pitch, const double* tb, int Vp,
                                               int nq, int lane, const double (&u)[3][2], double (&s)[3][2]) {
    const unsigned char* cx = reinterpret_cast<const unsigned char*>(tb);
    const unsigned char* cy = reinterpret_cast<const unsigned char*>(tb + Vp);
    const unsigned char* wj = reinterpret_cast<const unsigned char*>(tb + 2 * Vp);
#pragma unroll
    for (int r = 0; r < 3; ++r) s[r][0] = s[r][1] = 0.0;
    for_vectors(lane, nq, [&](int o) {
      const double2 c = at<double2>(cx, o), d = at<double2>(cy, o), w = at<double2>(wj, o);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double2 x = at<double2>(rows + r * pitch, o);
        const double dx0 = c.x - u[r][0], dy0 = d.x - u[r][1], dx1 = c.y - u[r][0], dy1 = d.y - u[r][1];
        const double q0v = dx0 * dx0 + dy0 * dy0, q1v = dx1 * dx1 + dy1 * dy1;
        const double a0 = w.x * x.x, a1 = w.y * x.y;
        s[r][0] = fma(q0v, a0, fma(q1v, a1, s[r][0]));                            // src/macros.f90:144-148, times 2
        s[r][1] = fma(sqrt_newton(q0v), a0, fma(sqrt_newton(q1v), a1, s[r][1]));  // src/compmu.f90:71-74
      }
    });
#pragma unroll
    for (int r = 0; r < 3; ++r) s[r][0] *= 0.5;
  }
};

// MACROS / COMPMU / GTEQNF per DG node from its velocity sums
// (src/macros.f90:126-154, src/compmu.f90:86-97, src/gteqnf.f90:28-37):
// s0 = n (before the 1e-20 test), (ux, uy), nd = n or 0, sp = the pressure
// sum over M/NA, sc = the mean-relative-speed sum; writes the node's
// moments, MU and the sweep's NFO parameters, returns MU.
template <class T>
__device__ __forceinline__ double node_epilogue(const CaseDev<T>& C, int node, double s0, double ux, double uy,
                                                double nd, double sp, double sc) {
  const double ps = sp * C.MM;
  // MU = sqrt(2) CT sigma n with CT = sc/n: the division and the product with
  // n cancel (0 where n < 1e-20)
  const double mu = (nd >= TINY_D) ? sqrt(2.0) * C.sigt * sc : 0.0;
  const int e = node / 3, i = node - 3 * (node / 3);
  ElemRec<T>& en = C.rec[e];
  // GTEQNF's parameters; FP64 in the expanded exponent form of the sweep
  // (ElemRec)
  if (ps >= TINY_D) {
    const double rho = C.MM * nd;
    const double b2 = rho / (2 * ps);
    const double a = nd * (b2 * (1.0 / PI_D));
    if (sizeof(T) == 4) {
      coef_set(en.A[i], a);
      coef_set(en.ex[i], -b2 * LOG2E_D);
      coef_set(en.ux[i], -ux);
      coef_set(en.uy[i], -uy);
    } else {
      coef_set(en.A[i], log(a) - b2 * (ux * ux + uy * uy));
      coef_set(en.ex[i], -b2);
      coef_set(en.ux[i], 2.0 * b2 * ux);
      coef_set(en.uy[i], 2.0 * b2 * uy);
    }
  } else {
    coef_set(en.A[i], sizeof(T) == 4 ? 0.0 : -INFINITY);
    coef_set(en.ex[i], 0.0);
    coef_set(en.ux[i], sizeof(T) == 4 ? -ux : 0.0);
    coef_set(en.uy[i], sizeof(T) == 4 ? -uy : 0.0);
  }
  coef_set(en.mu[i], mu);
  coef_set(en.mt[i], mu);
  C.nraw[node] = s0;
  C.disux[node] = ux;
  C.disuy[node] = uy;
  C.disps[node] = ps;
  C.mu[node] = mu;
  return mu;
}

// Sum over the L lanes of an aligned lane group (every lane gets the same
// bits: each butterfly level adds the same two operands in either order).
template <int L> __device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums over the warp of K values for each of three rows, row 0's left in
// lanes 0 to 7, row 1's in 8 to 15, row 2's in 16 to 31: the first two levels
// of the butterfly hand rows to lane groups, so each of the other three
// levels moves K values and not 3K (6K exchanges instead of 15K).
template <int K> __device__ __forceinline__ void row_sums(const double (&v)[3][K], int lane, double (&t)[K]) {
  const bool hi = (lane & 16) != 0, second = (lane & 24) == 8;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double x = (hi ? v[2][k] : v[0][k]) + __shfl_xor_sync(0xffffffffu, hi ? v[0][k] : v[2][k], 16);
    const double y = v[1][k] + __shfl_xor_sync(0xffffffffu, v[1][k], 16);
    t[k] = (second ? y : x) + __shfl_xor_sync(0xffffffffu, hi || second ? x : y, 8);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
}

// Moment kernel: persistent warps over the flattened row groups of all the
// cases; each warp takes R DG nodes (velocity rows) at a time, L = 32/R
// lanes per row, from a per-warp ring of stages filled by 1-D bulk copies,
// so f is read from HBM once for both passes.  ONE: a single case, passed
// as a kernel parameter, with its velocity tables staged in shared memory;
// otherwise the case table, with the tables read through L1 (they differ
// from case to case).  MU's maximum goes to the case's control block once
// per warp and case.  Up to 20 warps per CTA for a single case (at
// most 96 registers), 16 for the case table.
template <class T, int R, bool ONE>
__global__ void __launch_bounds__(ONE ? 640 : 512, 1)
    k_moments(BatchArgs<T> a, int total_groups, const __grid_constant__ CaseDev<T> one) {
  // R = 1, 2, 4: R rows of any elements per warp step, 32/R lanes per row;
  // R = 3: the three rows of one element per warp step, all 32 lanes on
  // each (the velocity tables loaded once for the three rows)
  constexpr bool ELEM = R == 3;
  constexpr int L = ELEM ? 32 : 32 / R;
  extern __shared__ __align__(128) unsigned char sm_raw[];
  const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform: the ring's addresses too
  const int grp = ELEM ? 0 : lane / L, sub = lane % L;
  const int nstage = a.mom_stages;
  // layout: [barriers][tables [mom_tables][Vp] (ONE)][rings: warp, stage, R rows]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm_raw) + warp * nstage;
  T* tb1 = reinterpret_cast<T*>(sm_raw + 128 * (((size_t)nwarp * nstage * 8 + 127) / 128));
  constexpr int NTB = mom_tables<T>(R);  // tables staged for a single case
  const size_t tbytes = ONE ? (NTB * (size_t)one.Vp * sizeof(T) + 127) / 128 * 128 : 0;
  const size_t stage_bytes = (size_t)R * a.mom_rowbytes;
  unsigned char* ring = reinterpret_cast<unsigned char*>(tb1) + tbytes + (size_t)warp * nstage * stage_bytes;
  if (ONE) {
    const uint4* src = reinterpret_cast<const uint4*>(one.tabs);
    for (int i = threadIdx.x; i < (int)(NTB * one.Vp * sizeof(T) / 16); i += blockDim.x)
      reinterpret_cast<uint4*>(tb1)[i] = src[i];
  }
  const int gw = blockIdx.x * nwarp + warp, stride = gridDim.x * nwarp;
  if (lane == 0) {
    for (int s = 0; s < nstage; ++s) mbar_init(&bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_launch_dependents();
  grid_wait();  // the state, the control blocks
  // lane 0: the rows of group g into stage s (none when the case is done)
  auto fill = [&](int s, int g) {
    const int c = ONE ? 0 : find_case(a.grp_off, a.ncases, g);
    const CaseDev<T>& C = ONE ? one : a.cases[c];
    const Ctrl* ctl = C.ctrl;
    const int r0 = (g - (ONE ? 0 : a.grp_off[c])) * R;
    const int nr = ctl->done ? 0 : min(R, 3 * C.E - r0);
    const T* f = C.f[ctl->cur];
    mbar_expect_tx(&bars[s], (unsigned)nr * C.rowbytes);
    for (int k = 0; k < nr; ++k)
      bulk_load(ring + (size_t)s * stage_bytes + (size_t)k * C.rowbytes, f + (size_t)(r0 + k) * C.Vp, C.rowbytes,
                &bars[s]);
  };
  if (lane == 0)
    for (int s = 0; s < nstage; ++s)
      if (gw + s * stride < total_groups) fill(s, gw + s * stride);
  uint32_t parity = 0;  // bit s: parity of stage s
  int s = 0;
  bool aborted = false;
  int mu_case = -1;
  double mumax = 0.0;
  // MU >= 0: the max of the bit patterns is the max of the values
  auto flush_mu = [&]() {
    const double m = warp_max(mumax);
    if (lane == 0 && mu_case >= 0 && m > 0.0)
      atomicMax(reinterpret_cast<unsigned long long*>(&(ONE ? one : a.cases[mu_case]).ctrl->maxmu),
                (unsigned long long)__double_as_longlong(m));
    mumax = 0.0;
  };
  // The lanes of a row's group all hold its sums; lane `kept` of the group
  // keeps them, and once every lane has a node the per-node epilogue (FP64
  // divisions, a logarithm, the stores) runs for all of them at once.  A node
  // at a time it was a third of the warp's instructions.
  constexpr int KEEP = ELEM ? 8 : L;
  int kept = 0, knode = -1;
  double k0 = 0, kux = 0, kuy = 0, ksp = 0, ksc = 0;
  auto flush_nodes = [&]() {
    if (knode >= 0)
      mumax = fmax(mumax, node_epilogue(ONE ? one : a.cases[mu_case], knode, k0, kux, kuy, k0 >= TINY_D ? k0 : 0.0,
                                        ksp, ksc));
    knode = -1;
    kept = 0;
  };
  int c = 0;
  for (int g = gw; g < total_groups; g += stride) {
    c = ONE ? 0 : find_case(a.grp_off, a.ncases, g);  // warp-uniform
    int ok = 1;
    if (lane == 0) ok = mbar_wait_bounded(&bars[s], (parity >> s) & 1) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) {
      aborted = true;
      break;
    }
    mbar_wait_bounded(&bars[s], (parity >> s) & 1);  // completed: returns at once
    parity ^= 1u << s;
    const CaseDev<T>& C = ONE ? one : a.cases[c];
    if (c != mu_case) {
      flush_nodes();
      flush_mu();
      mu_case = c;
    }
    const int node0 = (g - (ONE ? 0 : a.grp_off[c])) * R;
    const T* tb = ONE ? tb1 : C.tabs;
    const bool live0 = !C.ctrl->done;
    const int nql = live0 ? (int)(C.rowbytes / 16) : 0;
    // this lane's node and its sums: s0 = n, ux, uy (MACROS pass 1), sp, sc
    // (pass 2: pressure and COMPMU's mean relative speed)
    int node;
    double s0, ux, uy, sp, sc;
    if constexpr (ELEM) {
      const unsigned char* rows = ring + (size_t)s * stage_bytes;
      double m1[3][3], t1[3], m2[3][2], t2[2];
      ElemMath<T>::template pass1<ONE && sizeof(T) == 4>(rows, C.rowbytes, tb, C.Vp, nql, lane, m1);
      row_sums<3>(m1, lane, t1);
      s0 = t1[0];
      ux = uy = 0.0;
      if (s0 >= TINY_D) {  // src/macros.f90:126-134
        const double inv = 1.0 / s0;
        ux = t1[1] * inv;
        uy = t1[2] * inv;
      }
      T u[3][2];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        u[r][0] = __shfl_sync(0xffffffffu, (T)ux, 8 * r);
        u[r][1] = __shfl_sync(0xffffffffu, (T)uy, 8 * r);
      }
      ElemMath<T>::pass2(rows, C.rowbytes, tb, C.Vp, nql, lane, u, m2);
      row_sums<2>(m2, lane, t2);
      sp = t2[0];
      sc = t2[1];
      node = lane < 24 ? node0 + (lane >> 3) : 3 * C.E;  // lanes 16 to 23: row 2
    } else {
      node = node0 + grp;
      const T* row = reinterpret_cast<const T*>(ring + (size_t)s * stage_bytes + (size_t)grp * C.rowbytes);
      const int nqr = node < 3 * C.E ? nql : 0;
      double s1 = 0, s2 = 0;
      s0 = 0;
      RowMath<T>::pass1(row, tb, C.Vp, nqr, sub, L, s0, s1, s2);
      s0 = group_sum<L>(s0);
      s1 = group_sum<L>(s1);
      s2 = group_sum<L>(s2);
      ux = uy = 0;
      if (s0 >= TINY_D) {  // src/macros.f90:126-134
        const double inv = 1.0 / s0;
        ux = s1 * inv;
        uy = s2 * inv;
      }
      sp = sc = 0;
      RowMath<T>::pass2(row, tb, C.Vp, nqr, sub, L, ux, uy, sp, sc);
      sp = group_sum<L>(sp);
      sc = group_sum<L>(sc);
    }
    __syncwarp();
    // the rows are consumed: refill this stage with the group nstage ahead
    if (lane == 0) {
      const int nxt = g + nstage * stride;
      if (nxt < total_groups) {
        fence_proxy_async_smem();
        fill(s, nxt);
      }
    }
    if ((lane & (KEEP - 1)) == kept && live0 && node < 3 * C.E) {
      knode = node;
      k0 = s0;
      kux = ux;
      kuy = uy;
      ksp = sp;
      ksc = sc;
    }
    if (++kept == KEEP) flush_nodes();
    s = (s + 1 == nstage) ? 0 : s + 1;
  }
  if (aborted) {
    if (lane == 0) {
      (ONE ? one : a.cases[c]).ctrl->timeout = 1;
      for (int k = 0; k < nstage; ++k) mbar_wait_bounded(&bars[k], (parity >> k) & 1);
    }
    return;
  }
  flush_nodes();
  flush_mu();
}

// --------------------------------------------------------- wall flux ----
// FLUCON2 (src/flucon2.f90:134-233): one CTA (WALL_THREADS threads) per
// wall side of any case, its threads strided over the velocities, then a
// block sum (a warp per side left the loads of a side in a serial chain:
// ~37 us on the 200x100 channel's 40 wall sides).
constexpr int WALL_THREADS = 256;
template <class T> __global__ void __launch_bounds__(WALL_THREADS) k_wall(BatchArgs<T> a, int total_walls) {
  __shared__ double part[WALL_THREADS / 32];
  const int w = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (w >= total_walls) return;
  const int c = find_case(a.wall_off, a.ncases, w);
  const CaseDev<T>& C = a.cases[c];
  if (C.ctrl->done) return;  // the same for the whole CTA
  const WallSide ws = C.walls[w - a.wall_off[c]];
  const T* f = C.f[C.ctrl->cur];
  const T* f1 = f + ((size_t)ws.elem * 3 + ws.in1) * C.Vp;
  const T* f2 = f + ((size_t)ws.elem * 3 + ws.in2) * C.Vp;
  double s = 0;
  for (int v = threadIdx.x; v < C.V; v += WALL_THREADS) {
    const double test = C.cxD[v] * ws.anx + C.cyD[v] * ws.any;
    if (test > 0.0) s += fabs(test) * (0.5 * ((double)f1[v] + (double)f2[v])) * C.wjf[v];
  }
  s = warp_sum(s);
  if (lane == 0) part[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
#pragma unroll
    for (int k = 0; k < WALL_THREADS / 32; ++k) t += part[k];
    const double eta = t / ws.sumbottom;
    C.bEtaD[ws.bside] = eta;
    C.bwall[4 * (size_t)ws.bside + 3] = (T)((double)C.alpha * eta);
  }
}

// -------------------------------------------------------------- sweep ----
// DTE = min(CSAFE/maxMU, DTEc)  (src/alotim2.f90:10-15, src/advnce.f90:258-262)
__device__ __forceinline__ double step_dt(const Ctrl* c) {
  const double mx = c->maxmu, dtc = c->dtc;
  // well inside the collision limit the Courant limit is the smaller one: no
  // division in front of the kernel's first unit
  if (mx > 0.0 && mx * dtc < 0.899 && dtc < 1000000.0) return dtc;
  const double dtb = (mx > 0.0) ? 0.9 * (1.0 / mx) : 1000000.0;
  return fmin(dtb, dtc);
}

// ----------------------------------------------------------- residual ----
// GETRES + the residual bookkeeping (src/advnce.f90:385, 422-429) per case,
// one thread per case: the step's max and L2 residual into the history, the
// non-finite and convergence tests, the step counter and the buffer swap;
// the step's accumulators are cleared for the next step.  The sweep's last
// CTA runs it (or k_resid).
template <class T> __device__ __forceinline__ void resid_book(const CaseDev<T>& C, double mm, double sq) {
  Ctrl* c = C.ctrl;
  const int st = c->step;
  const double l2 = sqrt(sq);
  double* h = C.hist + 3 * (size_t)st;
  h[0] = mm;
  h[1] = l2;
  h[2] = step_dt(c);
  if (!isfinite(l2) || !isfinite(mm)) {
    c->nonfinite = 1;
    c->done = 1;
  }
  if (c->timeout) c->done = 1;
  if (c->ref == 0.0 && l2 > 0.0) c->ref = l2;
  c->acc_sq = 0.0;
  c->acc_max = 0.0;
  c->maxmu = 0.0;
  c->cur ^= 1;
  c->step = st + 1;
  if (c->step >= c->max_steps) c->done = 1;
  if (c->tol > 0.0 && l2 <= c->tol * c->ref) c->done = 1;
}
// Sweep geometry.  LPE = 8 lanes share an element, each with one 16-byte
// vector of velocities (4 FP32 or 2 FP64), so a warp works on EPW = 4
// elements at 32 (16) velocities and every row access -- global or shared --
// is a whole 128-byte line.  A tile is one such velocity segment of an
// element block and its halo: the rows of g = f - UMEAN, 128 bytes each, row
// r = 3*slot + i (block element j: slot j; halo element h: slot EB + h) at
// byte 128*r.  Eight lanes read a row through all 32 banks, so neither the
// own rows nor the neighbours' rows conflict.  A work unit is one block at
// consecutive velocity tiles: its element records, the halo's record heads
// and the halo list are staged in shared memory once per unit.
template <class T> struct SweepGeo {
  static constexpr int W = 16 / (int)sizeof(T);  // velocities per lane
  static constexpr int NP = W / 2 < 1 ? 1 : W / 2;  // pairs per lane
  static constexpr int LPE = 8;                  // lanes per element
  static constexpr int VT = W * LPE;             // velocities per tile
  static constexpr int EPW = 32 / LPE;           // elements of a warp at a time
  // block elements per lane group: their NFO and UMEAN stay in registers
  // between the phases (16 registers an element)
  static constexpr int ITERS = 2;
  static constexpr int threads(int EB) { return EB / (EPW * ITERS) * 32; }
  // resident CTAs per SM at 128 registers a thread (16 warps)
  static constexpr int min_ctas(int EB) { return 65536 / (128 * threads(EB)); }
  static constexpr int RW = (int)(sizeof(ElemRec<T>) / 16);                // record words
  static constexpr int HW = (REC_HEAD_VALUES * (int)sizeof(typename CoefOf<T>::type) + 15) / 16;  // head words
  // pitches in shared memory: odd numbers of 16-byte words, so that the four
  // records a warp reads at once fall on different banks
  static constexpr int RP = 16 * (RW | 1), HR = 16 * (HW | 1);
  static constexpr int TPU_MAX = 16;
  // rows of swtab: cx, cy, NFINF (and |c|^2 for the FP64 exponent)
  static constexpr int NTAB = sizeof(T) == 8 ? 4 : 3;
  static constexpr unsigned tile_bytes(int EB, int max_halo) { return tile_row(3 * (EB + max_halo)); }
  // velocity tables staged per unit: cx, cy (and |c|^2 for the FP64 exponent)
  static constexpr int NVT = sizeof(T) == 8 ? 3 : 2;
  // `bufs` tiles, records [EB], halo heads [max_halo], velocity tables
  // [NVT][TPU_MAX * VT], halo list [max_halo]
  static constexpr size_t smem(int EB, int max_halo, int bufs) {
    return (size_t)bufs * tile_bytes(EB, max_halo) + (size_t)EB * RP + (size_t)max_halo * HR +
           (size_t)NVT * TPU_MAX * ROW_BYTES + ((size_t)max_halo * 4 + 15) / 16 * 16;
  }
};

// 16-byte asynchronous copy global -> shared through L2 only (cp.async.cg).
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// exp of the NFO exponent: FP64 by Tang's table-driven method (exp_tang.h,
// about one ulp, `tab` the CTA's 2^(j/256) table); FP32 2^x from the SFU
// (ex2.approx, relative error ~2^-22; the FP32 coefficient carries the
// log2(e) factor, applied in FP64 by the moment kernel; no table).
template <class T> __device__ __forceinline__ T nfo_exp(T x, const double* tab);
template <> __device__ __forceinline__ double nfo_exp<double>(double x, const double* tab) {
  return exp_tang(x, tab);
}
template <> __device__ __forceinline__ float nfo_exp<float>(float x, const double*) {
  float p;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(x));
  return p;
}

// Pairs of velocities: FP32 on packed instructions (one issue slot for two
// values, each rounded as the scalar instruction would), FP64 scalar.
template <class T> struct Pair;
template <> struct Pair<float> { using type = float2; using vec = float4; };
template <> struct Pair<double> { using type = double2; using vec = double2; };
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 pdup(float a) { return make_float2(a, a); }
__device__ __forceinline__ double2 padd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 pmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 pfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 pdup(double a) { return make_double2(a, a); }
// a - b; FP32 as one packed fma(b, -1, a), the same rounding (negating a
// packed operand takes two instructions)
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ double2 psub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a record's coefficient as a pair and as a value
__device__ __forceinline__ float2 pdup(const CoefF& c) { return make_float2(c.x, c.y); }
__device__ __forceinline__ float pval(const CoefF& c) { return c.x; }
__device__ __forceinline__ double pval(double c) { return c; }
// the pairs of a 16-byte vector
__device__ __forceinline__ float2 pget(const float4& v, int h) { return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y); }
__device__ __forceinline__ double2 pget(const double2& v, int) { return v; }
__device__ __forceinline__ void pset(float4& v, int h, float2 p) {
  if (h) {
    v.z = p.x;
    v.w = p.y;
  } else {
    v.x = p.x;
    v.y = p.y;
  }
}
__device__ __forceinline__ void pset(double2& v, int, double2 p) { v = p; }

__device__ __forceinline__ float vec_at(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ double vec_at(const double2& v, int k) { return k == 0 ? v.x : v.y; }
template <class T> __device__ __forceinline__ typename Pair<T>::vec vld(const void* p) {
  return *reinterpret_cast<const typename Pair<T>::vec*>(p);
}
template <class T> __device__ __forceinline__ void vst(void* p, const typename Pair<T>::vec& v) {
  *reinterpret_cast<typename Pair<T>::vec*>(p) = v;
}
// Phase 1 of the sweep on one lane's velocities of an element's three rows:
// NFO (GTEQNF, src/gteqnf.f90:35-37) and UMEAN = 0.5*DTE*(div F -
// 1/3 sum_i MU_i (NFO_i - f_i)) with div F = sum_i (N_i,x cx + N_i,y cy) f_i
// (GETELC, src/getelc.f90:54-83); g = f - UMEAN, the value every edge flux
// and the volume term of this element use (src/getelc.f90:87-117,
// src/edgflxopt.f90:95-125), replaces f.  The staged record carries the
// gradients times 0.5*DTE and MU times -DTE/6 (sweep_scale).  FP32: NFO =
// A*2^(ex*|c-u|^2) with the SFU's 2^x; FP64: NFO = exp(a0 + a1*cx + a2*cy +
// ex*|c|^2) (the exponent expanded, three FMAs; c2 = |c|^2 per velocity).
template <class T>
__device__ __forceinline__ void sweep_p1(const ElemRec<T>& r, const double* etab, unsigned char* rows,
                                         const typename Pair<T>::vec& cxv, const typename Pair<T>::vec& cyv,
                                         const typename Pair<T>::vec& c2v, typename Pair<T>::vec (&q)[3],
                                         typename Pair<T>::vec& u) {
  using P = typename Pair<T>::type;
  typename Pair<T>::vec f[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) f[i] = vld<T>(rows + i * ROW_BYTES);
#pragma unroll
  for (int h = 0; h < SweepGeo<T>::NP; ++h) {
    const P cx = pget(cxv, h), cy = pget(cyv, h);
    P fi[3], um;
#pragma unroll
    for (int i = 0; i < 3; ++i) fi[i] = pget(f[i], h);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P qi;
      if constexpr (sizeof(T) == 8) {
        const P x = pfma(pdup(r.ux[i]), cx, pfma(pdup(r.uy[i]), cy, pfma(pdup(r.ex[i]), pget(c2v, h), pdup(r.A[i]))));
        qi.x = nfo_exp<T>(x.x, etab);
        qi.y = nfo_exp<T>(x.y, etab);
      } else {
        const P dx = padd(cx, pdup(r.ux[i])), dy = padd(cy, pdup(r.uy[i]));
        const P x = pmul(pdup(r.ex[i]), pfma(dx, dx, pmul(dy, dy)));
        qi.x = nfo_exp<T>(x.x, etab);
        qi.y = nfo_exp<T>(x.y, etab);
        qi = pmul(pdup(r.A[i]), qi);
      }
      pset(q[i], h, qi);
      const P t = psub(qi, fi[i]);
      um = i == 0 ? pmul(pdup(r.mu[0]), t) : pfma(pdup(r.mu[i]), t, um);
    }
    const P sx = pfma(pdup(r.gx[2]), fi[2], pfma(pdup(r.gx[1]), fi[1], pmul(pdup(r.gx[0]), fi[0])));
    const P sy = pfma(pdup(r.gy[2]), fi[2], pfma(pdup(r.gy[1]), fi[1], pmul(pdup(r.gy[0]), fi[0])));
    um = pfma(sx, cx, pfma(sy, cy, um));
    pset(u, h, um);
#pragma unroll
    for (int i = 0; i < 3; ++i) pset(f[i], h, psub(fi[i], um));
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) vst<T>(rows + i * ROW_BYTES, f[i]);
}

// The step's factors of a staged record, applied to its 16-byte words (two
// coefficients) by the lane that copied them: 0.5*DTE to the gradients (words
// 0 to 2), -DTE/6 to MU (words 9, 10), DTE to MT and MM (words 11 to 13); the
// other words are left alone.
__device__ __forceinline__ bool sweep_scaled(int word) { return word < 3 || (word >= 9 && word < 14); }
template <class T> __device__ __forceinline__ void sweep_scale(unsigned char* word, T s) {
  typename Pair<T>::vec v = vld<T>(word);
#pragma unroll
  for (int h = 0; h < SweepGeo<T>::NP; ++h) pset(v, h, pmul(pget(v, h), pdup(s)));
  vst<T>(word, v);
}

// max that keeps a NaN operand (max.NaN): the residual's "change the
// unknown receives" must carry a non-finite update into the L2 sum
__device__ __forceinline__ float fmax_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Adds the per-warp residual partials (max |d|, sum of squares) to a case's
// accumulators.
template <int NW>
__device__ __forceinline__ void resid_add(Ctrl* ctrl, const double* red_m, const double* red_s) {
  double mm = 0, ss = 0;
  for (int w = 0; w < NW; ++w) {
    mm = fmax(mm, red_m[w]);
    ss += red_s[w];
  }
  atomicAdd(&ctrl->acc_sq, ss);
  atomicMax(reinterpret_cast<unsigned long long*>(&ctrl->acc_max), (unsigned long long)__double_as_longlong(mm));
}

// Persistent sweep kernel.  Work units are (block b, group of `tpu` velocity
// tiles) with b fastest, handed out in order (the first by blockIdx, the
// rest from a device counter), so the CTAs running at one moment cover
// neighbouring blocks at the same velocities and the halo rows they read are
// L2 hits.  Per unit the block's element records, the halo's record heads and
// the unit's velocities are staged in shared memory; per tile
//  * the rows of every block and halo element are copied to the tile by the
//    lanes that will work on them (cp.async, a tile ahead: they wait for
//    their own copies only);
//  * phase 1: UMEAN and g = f - UMEAN, which replaces f in the tile; a block
//    element's NFO and UMEAN stay in the registers of the lanes that update
//    it;
//  * phase 2, the same lanes update the element: the volume term
//    (src/getelc.f90:87-117) and the edge fluxes gathered per element from
//    the tile (EDGFLXOPT src/edgflxopt.f90:95-125; an outflow side reads the
//    element itself), the wall sides' fluxes (GETBOU
//    src/getbou.f90:142-281), GETINC/CMMINC, ADTHEM and INFLOW; the new rows
//    go to global memory as whole lines.
// With two tile buffers one barrier per tile is enough (between its phases:
// a warp past it has left the previous tile, whose buffer the copies of the
// next one overwrite); a mesh whose halo leaves room for one buffer only
// takes a second barrier after phase 2.
// ONE: a single case passed as a kernel parameter (its fields come from the
// constant bank, no registers); otherwise the case table.
// Upwinding: the own value is taken where SC = n.c > 0.  The reference takes
// it where SC > 0 for the ISIDE(3) element and SC >= 0 for the other; the
// two differ only at SC = 0, where the flux SC*value is zero either way.
//
// Why this mapping.  FP32 issues 486 warp instructions per 128 (element,
// velocity) pairs, halo included; two lanes per element at 8 velocities each,
// 64-byte swizzled rows and scalar arithmetic took 760.  What went: half of
// the FMA-pipe issue slots (packed pairs), the duplication of coefficients
// (the records hold them as pairs) and the swizzle's index arithmetic, the
// staging of the new rows through the tile, and the neighbour gather's bank
// conflicts (2.0e7 -> 0.3e7 per launch).  200x100 channel, 24x48 velocities
// (1.375e8 DOFs): FP32 0.394 -> 0.293 ms, FP64 0.945 -> 0.742.  Bound (FP32,
// ncu): latency at 16 warps per SM (128 registers), issue active 0.52, stalls
// per issue wait 1.2, short-scoreboard and barrier 0.9 each, math-pipe 0.9;
// FMA pipe 0.41 and shared-memory wavefronts 0.62 of their peaks.  Measured
// and not kept: one element per lane group and 16 warps per 64 elements
// (FP32 0.372, FP64 0.817), four per group in FP64 (1.04), FP64 at 168
// registers (0.840), coefficients duplicated in registers (0.387), f loaded
// straight into registers at the start of phase 1 (0.387), one tile buffer
// and three CTAs at 80 registers (FP32 0.358), the wall records staged in
// shared memory (FP32 0.295, FP64 0.788).  At 128 registers FP32 with IMMAT =
// 1 does not spill; the others do (bytes of stores per thread, a single case /
// a batch: FP64 76 to 80 / 124, FP64 with IMMAT = 0 112 / 120, FP32 with
// IMMAT = 0, which reads the residual tables in the update, 168 / 84).
template <class T, int EB, int IMMAT, bool ONE>
__global__ void __launch_bounds__(SweepGeo<T>::threads(EB), SweepGeo<T>::min_ctas(EB))
    k_sweep(BatchArgs<T> a, int total_units, const __grid_constant__ CaseDev<T> one) {
  using G = SweepGeo<T>;
  using P = typename Pair<T>::type;
  using VecT = typename Pair<T>::vec;
  constexpr int W = G::W, NP = G::NP, VT = G::VT, RW = G::RW, RP = G::RP, HW = G::HW, HR = G::HR;
  constexpr int ITERS = G::ITERS, EPW = G::EPW;
  constexpr int NT = G::threads(EB), NW = NT / 32;
  static_assert(NW * EPW * ITERS == EB, "whole warps");
  extern __shared__ __align__(128) unsigned char sm_raw[];
  // the next unit, handed from thread 0 to the CTA: two slots used in turn,
  // so thread 0 never overwrites the slot another warp may still be reading
  // (a unit of a finished case has no barrier of its own: with one slot,
  // thread 0 could loop round and replace the value before a slow warp read
  // it, and the warps would then disagree on the unit and on the barriers)
  __shared__ int s_unit[2], s_last;
  __shared__ double red_m[NW], red_s[NW];
  // FP64: the 2^(j/256) table of the NFO exp (one entry for FP32, unused)
  __shared__ double etab[sizeof(T) == 8 ? EXP_TAB : 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub = lane / G::LPE, l8 = tid & (G::LPE - 1);
  if (sizeof(T) == 8)
    for (int i = tid; i < EXP_TAB; i += NT) etab[i] = a.ctl->etab[i];
  const unsigned tile_bytes = G::tile_bytes(EB, a.max_halo);
  const bool two = a.sweep_bufs > 1;
  unsigned char* const recs = sm_raw + (two ? 2 : 1) * tile_bytes;  // pitch RP
  unsigned char* const hrec = recs + EB * RP;                       // pitch HR
  unsigned char* const vtab = hrec + (size_t)a.max_halo * HR;       // [NVT][TPU_MAX] rows
  int* const hl = reinterpret_cast<int*>(vtab + G::NVT * G::TPU_MAX * ROW_BYTES);  // the halo's elements
  const int j0 = warp * EPW + sub;  // the lane group's block elements: j0 + it*NW*EPW
  if (tid < ROW_BYTES / 4) {  // the tiles' rows of zeros
    reinterpret_cast<float*>(sm_raw)[tid] = 0.f;
    if (two) reinterpret_cast<float*>(sm_raw + tile_bytes)[tid] = 0.f;
  }

  int unit = blockIdx.x, c = 0, iter = 0;
  int gk = 0;  // tiles this CTA has started
  // residual partials of the thread's values: a single case adds them to its
  // control block once per CTA (after the last unit), a batch once per unit
  double rmax = 0.0, rsq = 0.0;
  // a single case's control values, the same for every unit
  int cur = 0;
  double dtd = 0.0;
  bool active = false;
  auto control = [&](const Ctrl* ctl) {
    active = !ctl->done;
    cur = ctl->cur;
    dtd = step_dt(ctl);
  };
  grid_launch_dependents();
  grid_wait();  // the moments and walls, the control blocks, the unit counter
  if (ONE) control(one.ctrl);
  // the unit after this one, drawn ahead so the atomic's latency is hidden
  int next = (tid == 0 && unit < total_units) ? (int)gridDim.x + atomicAdd(&a.ctl->sweep_next, 1) : 0;
  while (unit < total_units) {
    c = ONE ? 0 : find_case(a.unit_off, a.ncases, unit);
    const CaseDev<T>& C = ONE ? one : a.cases[c];
    if (!ONE) control(C.ctrl);  // the same for every thread
    if (active) {
      const int lu = unit - (ONE ? 0 : a.unit_off[c]);
      const int b = lu % C.nblocks, vg = lu / C.nblocks;
      const int e0 = b * EB, nb = min(EB, C.E - e0);
      // the halo: its count, and the first entries each thread needs before
      // the count is there (two loads in flight instead of one after the
      // other; entries past the count are valid element numbers)
      const int* __restrict__ hrow = C.halo + (size_t)b * C.hp;
      const int nh = hrow[0];
      constexpr int NHW = NT / 16;  // half-warps
      constexpr int PRE_H = 2, PRE_R = 2;
      int idh[PRE_H], idr[PRE_R];
#pragma unroll
      for (int x = 0; x < PRE_H; ++x) idh[x] = hrow[min(1 + (tid >> 4) + x * NHW, C.hp - 1)];
#pragma unroll
      for (int x = 0; x < PRE_R; ++x) idr[x] = hrow[min(1 + j0 + x * NW * EPW, C.hp - 1)];
      int vt0, ntl;
      sweep_group(C, vg, vt0, ntl);
      const T dt = (T)dtd;
      const T* __restrict__ fo = C.f[cur];
      T* __restrict__ fnw = C.f[cur ^ 1];
      const unsigned pitch = (unsigned)C.Vp * (unsigned)sizeof(T);
      unsigned own[ITERS];  // first rows of the lane group's elements
#pragma unroll
      for (int it = 0; it < ITERS; ++it) own[it] = 3u * (unsigned)(e0 + min(j0 + it * NW * EPW, nb - 1));
      // Copies of tile vt's rows into a buffer by the lanes that will work on
      // them in phase 1 (so a lane waits for its own copies only): the lane
      // group's block elements (past the end of the mesh the last one again)
      // and its share of the halo.
      auto issue = [&](int vt, unsigned char* buf, auto first) {
        constexpr bool FIRST = decltype(first)::value;  // the unit's first tile: hl is not there yet
        const unsigned char* src = reinterpret_cast<const unsigned char*>(fo + (size_t)vt * VT + l8 * W);
        auto copy3 = [&](int slot, unsigned row) {
#pragma unroll
          for (int i = 0; i < 3; ++i)
            cp_async16(buf + tile_row(3 * slot + i) + 16 * l8, src + (unsigned long long)(row + i) * pitch);
        };
#pragma unroll
        for (int it = 0; it < ITERS; ++it) copy3(j0 + it * NW * EPW, own[it]);
        if constexpr (FIRST) {
#pragma unroll
          for (int x = 0; x < PRE_R; ++x)
            if (j0 + x * NW * EPW < nh) copy3(EB + j0 + x * NW * EPW, 3u * (unsigned)idr[x]);
        }
#pragma unroll 1
        for (int h = j0 + (FIRST ? PRE_R : 0) * NW * EPW; h < nh; h += NW * EPW)
          copy3(EB + h, 3u * (unsigned)(FIRST ? hrow[1 + h] : hl[h]));
        cp_async_commit();
      };
      // unit prologue, all of it asynchronous: the block's element records
      // (a warp per record, a lane per word), the halo's record heads (a
      // half-warp each) and the unit's velocities, then the first tile's
      // rows; the records are scaled by the step's factors as they land, by
      // the lanes that copied them
      {
        const uint4* src = reinterpret_cast<const uint4*>(C.rec + e0);
        if (lane < RW)
#pragma unroll 4
          for (int j = warp; j < nb; j += NW) cp_async16(recs + j * RP + 16 * lane, src + j * RW + lane);
        const int hw = tid & 15, hs = tid >> 4;
        if (hw < HW) {
#pragma unroll
          for (int x = 0; x < PRE_H; ++x)
            if (hs + x * NHW < nh)
              cp_async16(hrec + (hs + x * NHW) * HR + 16 * hw, reinterpret_cast<const uint4*>(C.rec + idh[x]) + hw);
#pragma unroll 1
          for (int s = hs + PRE_H * NHW; s < nh; s += NHW)
            cp_async16(hrec + s * HR + 16 * hw, reinterpret_cast<const uint4*>(C.rec + hrow[1 + s]) + hw);
        }
        for (int w = tid; w < G::NVT * ntl * G::LPE; w += NT) {
          const int t = w / (ntl * G::LPE), x = w - t * ntl * G::LPE;
          cp_async16(vtab + t * G::TPU_MAX * ROW_BYTES + 16 * x,
                     C.swtab + (size_t)(t == 2 ? 3 : t) * C.Vp + (size_t)vt0 * VT + (size_t)x * W);
        }
        cp_async_commit();
        issue(vt0, sm_raw + (two ? (gk & 1) * tile_bytes : 0), std::true_type());
        for (int s = tid; s < nh; s += NT) hl[s] = hrow[1 + s];
        cp_async_wait<1>();
        const T dth = (T)(0.5 * dtd), mdt6 = (T)(-0.5 * dtd / 3.0);
        if (sweep_scaled(lane)) {
          const T sc = lane < 3 ? dth : lane < 11 ? mdt6 : dt;
#pragma unroll 4
          for (int j = warp; j < nb; j += NW) sweep_scale<T>(recs + j * RP + 16 * lane, sc);
        }
        if (hw < HW && sweep_scaled(hw)) {
          const T sc = hw < 3 ? dth : mdt6;
          for (int s = hs; s < nh; s += NHW) sweep_scale<T>(hrec + s * HR + 16 * hw, sc);
        }
        __syncthreads();
        // the wall records of the lane group's elements into L1
        if (l8 < 3)
#pragma unroll
          for (int it = 0; it < ITERS; ++it) {
            const int bs = reinterpret_cast<const ElemRec<T>*>(recs + min(j0 + it * NW * EPW, nb - 1) * RP)->bside[l8];
            if (bs >= 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(C.bwall + 4 * (size_t)bs));
          }
      }

      for (int k = 0; k < ntl; ++k, ++gk) {
        unsigned char* const tl8 = sm_raw + (two ? (gk & 1) * tile_bytes : 0) + 16 * l8;
        const int v0 = (vt0 + k) * VT + l8 * W;  // the lane's first velocity
        const unsigned char* vt = vtab + k * ROW_BYTES + 16 * l8;
        const VecT cxv = vld<T>(vt), cyv = vld<T>(vt + G::TPU_MAX * ROW_BYTES),
                   c2v = vld<T>(vt + (G::NVT - 1) * G::TPU_MAX * ROW_BYTES);  // |c|^2 (FP64)
        cp_async_wait<0>();

        // ---- phase 1: the lane group's block elements and its share of
        // the halo
        VecT q[ITERS][3], u[ITERS];
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
          const int j = j0 + it * NW * EPW;
          sweep_p1<T>(*reinterpret_cast<const ElemRec<T>*>(recs + min(j, nb - 1) * RP), etab, tl8 + tile_row(3 * j), cxv, cyv, c2v, q[it], u[it]);
        }
#pragma unroll 1
        for (int h = j0; h < nh; h += NW * EPW) {
          VecT qh[3], uh;
          sweep_p1<T>(*reinterpret_cast<const ElemRec<T>*>(hrec + (size_t)h * HR), etab,
                      tl8 + tile_row(3 * (EB + h)), cxv, cyv, c2v, qh, uh);
        }
        __syncthreads();
        if (two && k + 1 < ntl) issue(vt0 + k + 1, sm_raw + ((gk + 1) & 1) * tile_bytes, std::false_type());

        // ---- phase 2: the update of the lane group's block elements
        const bool whole = (vt0 + k + 1) * VT <= C.V;  // no velocity of the tile past V
        T rmt = (T)0;
        P sqt = pdup((T)0);
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
          const int j = j0 + it * NW * EPW;
          const bool live = j < nb;  // past the end of the mesh: nothing is written
          const ElemRec<T>& r = *reinterpret_cast<const ElemRec<T>*>(recs + min(j, nb - 1) * RP);
          const int flags = r.flags;
          P rhs[3][NP], sgm[NP], g[3][NP];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const VecT gv = vld<T>(tl8 + tile_row(3 * j + i));
#pragma unroll
            for (int h = 0; h < NP; ++h) g[i][h] = pget(gv, h);
          }
#pragma unroll
          for (int h = 0; h < NP; ++h) sgm[h] = padd(padd(g[0][h], g[1][h]), g[2][h]);
          // Edge fluxes (EDGFLXOPT, src/edgflxopt.f90:95-125): RHS_p -=
          // AL*SC*(2 u_p + u_q), RHS_q -= AL*SC*(u_p + 2 u_q), (u_p, u_q)
          // the element's own values where AL*SC > 0, the source's otherwise.
          // The node opposite the edge takes GETELC's volume term RHS_i =
          // AREA/3 (N_i,x cx + N_i,y cy) sum(g) (src/getelc.f90:87-117): for
          // P1, AREA/3 grad N_i = -(EL/6) n of that edge.  -AL*SC is formed,
          // so that every term is one fused multiply-add.
#pragma unroll
          for (int k2 = 0; k2 < 3; ++k2) {
            const int p = k2, qn = (k2 + 1) % 3, op = (k2 + 2) % 3;
            const VecT gpv = vld<T>(tl8 + r.off[k2][0]), gqv = vld<T>(tl8 + r.off[k2][1]);
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              const P ms = pfma(pdup(r.en[k2][0]), pget(cxv, h), pmul(pdup(r.en[k2][1]), pget(cyv, h)));  // -AL*SC
              const P gp = pget(gpv, h), gq = pget(gqv, h);
              P up, uq;
              up.x = ms.x < (T)0 ? g[p][h].x : gp.x;
              up.y = ms.y < (T)0 ? g[p][h].y : gp.y;
              uq.x = ms.x < (T)0 ? g[qn][h].x : gq.x;
              uq.y = ms.y < (T)0 ? g[qn][h].y : gq.y;
              const P fp = pfma(pdup((T)2), up, uq), fq = pfma(pdup((T)2), uq, up);
              if (k2 == 0) {
                rhs[p][h] = pmul(ms, fp);
                rhs[qn][h] = pmul(ms, fq);
                rhs[op][h] = pmul(ms, sgm[h]);
              } else {
                rhs[p][h] = pfma(ms, fp, rhs[p][h]);
                rhs[qn][h] = pfma(ms, fq, rhs[qn][h]);
                rhs[op][h] = pfma(ms, sgm[h], rhs[op][h]);
              }
            }
          }
          // ALPHA < 1: bit 3*w + i marks node i at velocity v0 + w as deferred
          // (its update gets the specular part in k_wspec)
          unsigned dmask = 0u;
          if (flags & 0x1f8) {
            // Wall sides: molecules leaving the wall (src/getbou.f90:189-255)
            // carry the diffuse part ALPHA*ETA*Mw here, the specular part
            // (1-ALPHA)*Rf in k_wspec; inflow sides: no flux.  The edge loop
            // has added the element's own values where AL*SC > 0 and nothing
            // elsewhere: the difference is added.
            const bool spec = C.spec != 0;
            // one edge at a time by its number, so that lanes whose wall is a
            // different local edge go together (and the code is there once)
            for (int em = ((flags >> 3) | (flags >> 6)) & 7; em != 0; em &= em - 1) {
              const int k2 = __ffs(em) - 1;
              const bool inflow = (flags & (FLAG_INFLOW_EDGE0 << k2)) != 0;
              const T wnx = pval(r.en[k2][0]), wny = pval(r.en[k2][1]);  // -AL*n of the side
              const int bs = inflow ? 0 : r.bside[k2];
              const VecT* wr = reinterpret_cast<const VecT*>(C.bwall + 4 * (size_t)bs);
              T w4[4];
              if constexpr (sizeof(T) == 4) {
                const VecT a4 = wr[0];
                w4[0] = a4.x, w4[1] = a4.y, w4[2] = a4.z, w4[3] = a4.w;
              } else {
                const VecT a2 = wr[0], b2 = wr[1];
                w4[0] = a2.x, w4[1] = a2.y, w4[2] = b2.x, w4[3] = b2.y;
              }
              // with the specular part, the wall branch is taken where the
              // host's FP64 TEST < 0 (the items of k_wspec are built from
              // it): one bit per velocity
              const bool sp = spec && !inflow;
              const unsigned tb = sp ? C.rf_bits[(size_t)bs * C.rf_words + (v0 >> 5)] >> (v0 & 31) : 0u;
              const unsigned nodes = k2 == 0 ? 3u : k2 == 1 ? 6u : 5u;
              auto wall = [&](int w, T cx, T cy, T gp, T gq, T& rp, T& rq) {
                const T ms = wnx * cx + wny * cy;  // -AL*SC, as in the edge loop
                const bool mine = sp ? !((tb >> w) & 1u) : ms <= (T)0;
                T up = gp, uq = gq;
                if (inflow) {
                  up = uq = (T)0;
                } else if (!mine) {
                  const T dx = cx - w4[0], dy = cy - w4[1];
                  up = uq = w4[3] * nfo_exp<T>(w4[2] * (dx * dx + dy * dy), etab);
                  if (sp) dmask |= nodes << (3 * w);
                }
                if (ms < (T)0) {
                  up -= gp;
                  uq -= gq;
                }
                rp = ms * ((T)2 * up + uq);
                rq = ms * (up + (T)2 * uq);
              };
#pragma unroll
              for (int h = 0; h < NP; ++h) {
                const P cx = pget(cxv, h), cy = pget(cyv, h);
                const P gp = k2 == 0 ? g[0][h] : k2 == 1 ? g[1][h] : g[2][h];
                const P gq = k2 == 0 ? g[1][h] : k2 == 1 ? g[2][h] : g[0][h];
                P rp, rq;
                wall(2 * h, cx.x, cy.x, gp.x, gq.x, rp.x, rq.x);
                wall(2 * h + 1, cx.y, cy.y, gp.y, gq.y, rp.y, rq.y);
                const P z = pdup((T)0);
                rhs[0][h] = padd(rhs[0][h], k2 == 0 ? rp : k2 == 2 ? rq : z);
                rhs[1][h] = padd(rhs[1][h], k2 == 1 ? rp : k2 == 0 ? rq : z);
                rhs[2][h] = padd(rhs[2][h], k2 == 2 ? rp : k2 == 1 ? rq : z);
              }
            }
          }
          // GETINC / CMMINC, ADTHEM (f >= 0), INFLOW and the residual.  Plain:
          // every value of the lane is updated and counted; otherwise those
          // past V (which stay zero), of nodes INFLOW resets and deferred
          // ones are left out of the residual.
          P sq = pdup((T)0);
          VecT out[3];
          auto finish = [&](auto plain) {
            constexpr bool PLAIN = decltype(plain)::value;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              T cmx = (T)0, cmn = (T)0;
              if (IMMAT == 0) {
                cmx = C.cmax[3 * (e0 + min(j, nb - 1)) + i];
                cmn = C.cmin[3 * (e0 + min(j, nb - 1)) + i];
              }
#pragma unroll
              for (int h = 0; h < NP; ++h) {
                const P f = padd(g[i][h], pget(u[it], h));
                const P cdt = pmul(pdup(r.mt[i]), psub(pget(q[it][i], h), f));  // COLL*DTE
                const P d = pfma(pdup(r.mm[i]), rhs[i][h], cdt);
                P rr, ch, fn = padd(f, d);
                if (IMMAT == 1) {
                  rr.x = fabs(d.x);
                  rr.y = fabs(d.y);
                } else {
                  rr.x = fmax((rhs[i][h].x >= (T)0 ? cmx : cmn) * (rhs[i][h].x * dt) + cdt.x, (T)0);
                  rr.y = fmax((rhs[i][h].y >= (T)0 ? cmx : cmn) * (rhs[i][h].y * dt) + cdt.y, (T)0);
                }
                // L2 residual: the change the unknown receives (-f where
                // the clip applies, i.e. where d < -f; none at inflow-reset
                // nodes); a non-finite d or f reaches the sum
                if constexpr (sizeof(T) == 4) {
                  ch.x = fmax_nan(d.x, -f.x);
                  ch.y = fmax_nan(d.y, -f.y);
                } else {
                  ch.x = fn.x < (T)0 ? -f.x : d.x;
                  ch.y = fn.y < (T)0 ? -f.y : d.y;
                }
                fn.x = fmax(fn.x, (T)0);
                fn.y = fmax(fn.y, (T)0);
                if constexpr (!PLAIN) {
                  auto value = [&](int w, T dd, T xx, T cc, T& rrr, T& chh, T& ff) {
                    const bool past = v0 + w >= C.V, def = ((dmask >> (3 * w + i)) & 1u) != 0 && !past;
                    if (past) ff = (T)0;
                    if (past || def) rrr = (T)0;
                    if (past || def || (flags & (1 << i))) chh = (T)0;
                    if (def && live) {
                      // k_wspec adds the specular part, clips and counts the
                      // residual
                      const size_t o = ((size_t)r.wslot * 3 + i) * C.Vp + v0 + w;
                      C.wd[o] = IMMAT == 1 ? dd : xx * dt;
                      if (IMMAT == 0) C.wd[(size_t)C.n_spec_slots * 3 * C.Vp + o] = cc;
                    }
                  };
                  value(2 * h, d.x, rhs[i][h].x, cdt.x, rr.x, ch.x, fn.x);
                  value(2 * h + 1, d.y, rhs[i][h].y, cdt.y, rr.y, ch.y, fn.y);
                }
                rmt = fmax(rmt, fmax(rr.x, rr.y));
                sq = pfma(ch, ch, sq);
                pset(out[i], h, fn);
              }
            }
          };
          if (whole && (flags & 7) == 0 && dmask == 0u) {
            finish(std::true_type());
          } else {
            finish(std::false_type());
            if (flags & 7) {
              const VecT nf = vld<T>(C.nfinf + v0);  // zero past V
#pragma unroll
              for (int i = 0; i < 3; ++i)
                if (flags & (1 << i)) out[i] = nf;
            }
          }
          if (live) {
            sqt = padd(sqt, sq);
            unsigned char* dst = reinterpret_cast<unsigned char*>(fnw + v0);
#pragma unroll
            for (int i = 0; i < 3; ++i) vst<T>(dst + (unsigned long long)(own[it] + i) * pitch, out[i]);
          }
        }
        rmax = fmax(rmax, (double)rmt);
        rsq += (double)sqt.x + (double)sqt.y;
        if (!two && k + 1 < ntl) {
          __syncthreads();
          issue(vt0 + k + 1, sm_raw, std::false_type());
        }
      }
      // a batch: the unit's residual, per warp
      if (!ONE) {
        rmax = warp_max(rmax);
        rsq = warp_sum(rsq);
        if ((tid & 31) == 0) {
          red_m[warp] = rmax;
          red_s[warp] = rsq;
        }
        rmax = rsq = 0.0;
      }
    }
    // every thread is past phase 2 of the unit's last tile: (a batch) add the
    // unit's residual to its case (the sum of squares can differ in its last
    // bits between runs: the order of the atomics varies); the records and
    // the halo list may be replaced
    if (tid == 0) s_unit[iter & 1] = next;
    __syncthreads();
    if (!ONE && active && tid == 0) resid_add<NW>(C.ctrl, red_m, red_s);
    unit = s_unit[iter & 1];
    ++iter;
    if (tid == 0 && unit < total_units) next = (int)gridDim.x + atomicAdd(&a.ctl->sweep_next, 1);
  }
  // a single case: the CTA's residual (only a CTA that updated values; the
  // case's flag is the same for all of them)
  if (ONE && gk > 0) {
    rmax = warp_max(rmax);
    rsq = warp_sum(rsq);
    if ((tid & 31) == 0) {
      red_m[warp] = rmax;
      red_s[warp] = rsq;
    }
    __syncthreads();
    if (tid == 0) resid_add<NW>(one.ctrl, red_m, red_s);
  }
  // the last CTA to get here: every residual has been added and every unit
  // drawn, so the counters go back to zero and (fuse_resid) the cases' step is
  // booked here; as a launch of its own that took 2.5 us of each step
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(&a.ctl->sweep_done, 1) == (int)gridDim.x - 1;
    if (s_last) {
      __threadfence();
      a.ctl->sweep_next = 0;
      a.ctl->sweep_done = 0;
    }
  }
  if (!a.fuse_resid) return;
  if (ONE) {
    if (tid != 0 || !s_last || one.ctrl->done) return;
    resid_book(one, __ldcg(&one.ctrl->acc_max), __ldcg(&one.ctrl->acc_sq));
  } else {
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int k = tid; k < a.ncases; k += NT) {
      const CaseDev<T>& C = a.cases[k];
      if (!C.ctrl->done) resid_book(C, __ldcg(&C.ctrl->acc_max), __ldcg(&C.ctrl->acc_sq));
    }
  }
}

// ------------------------------------------------ specular wall part ----
// GETBOU's specular part for ALPHA < 1 (src/getbou.f90:189-255): a molecule
// leaving wall side k of element e at velocity v carries UNSID =
// (1-ALPHA)*Rf + ALPHA*ETA*Mw with Rf = (ZD2*f(I1) + ZD1*f(I2)) / (ZD1 +
// ZD2) of the element's own nodes at the mirrored grid velocities.  The
// reference reads f(I) from DISNF while its velocity loop updates it in
// place: the new value for I < v, the old one for I > v.  The sweep has
// applied the diffuse part and stored the deferred nodes' partial update
// (wd); the specular part is linear in RHS: with IMMAT = 1, DELUN +=
// MMAT*DTE*dRHS with dRHS the edge term of (1-ALPHA)*Rf; with IMMAT = 0
// CMMINC (src/cmminc.f90:22-41) on RHS*DTE + dRHS*DTE, its residual from the
// CMMAT row's largest or smallest entry; then ADTHEM's clip, INFLOW's reset
// and the residual.  seq = 0: the items whose mirrored velocities include no earlier
// deferred one, a thread each; seq = 1: the others, after the parallel ones, a
// warp per wall element: level by level (an item reads new values of earlier
// levels only), the items of a level side by side.  A thread per wall element
// took them one by one in velocity order, a chain of dependent loads an item
// (12x12 cavity, ALPHA 0.9, 18x18 velocities, FP64: step 212 -> 43 us; FP32
// 172 -> 39; 32x32 at 16x16, FP64: 203 -> 49).
template <class T> __global__ void __launch_bounds__(256) k_wspec(const __grid_constant__ CaseDev<T> C, int seq) {
  if (C.ctrl->done) return;
  const T dt = (T)step_dt(C.ctrl);
  const int cur = C.ctrl->cur;
  const T* __restrict__ fo = C.f[cur];
  T* fnw = C.f[cur ^ 1];
  const T om = (T)1 - C.alpha;
  double mx = 0.0, sq = 0.0;
  auto item = [&](int it) {
    const int s = it / C.V, v = it - s * C.V;
    const int e = C.welem[s];
    const ElemRec<T>& r = C.rec[e];
    const T cx = C.cx[v], cy = C.cy[v];
    T drhs[3] = {(T)0, (T)0, (T)0};
    unsigned mask = 0u;
    auto F = [&](int node, int I) {
      const size_t o = ((size_t)e * 3 + node) * C.Vp + I;
      return I < v ? fnw[o] : fo[o];
    };
    for (int k = 0; k < 3; ++k) {
      if (!(r.flags & (8 << k))) continue;
      const size_t o = ((size_t)C.rside[r.bside[k]] * C.V + v) * 2;
      const int i1 = C.rf_i[o], i2 = C.rf_i[o + 1];
      if (i1 < 0) continue;
      const T zd1 = C.rf_z[o], zd2 = C.rf_z[o + 1];
      const int p = k, q = (k + 1) % 3;
      const T dp = om * ((zd2 * F(p, i1) + zd1 * F(p, i2)) / (zd1 + zd2));
      const T dq = om * ((zd2 * F(q, i1) + zd1 * F(q, i2)) / (zd1 + zd2));
      const T as = -(pval(r.en[k][0]) * cx + pval(r.en[k][1]) * cy);  // AL * (n.c)
      drhs[p] -= as * ((T)2 * dp + dq);
      drhs[q] -= as * (dp + (T)2 * dq);
      mask |= (1u << p) | (1u << q);
    }
    for (int i = 0; i < 3; ++i) {
      if (!((mask >> i) & 1u)) continue;
      const size_t o = ((size_t)e * 3 + i) * C.Vp + v;
      const size_t od = ((size_t)s * 3 + i) * C.Vp + v;
      T d, rr;
      if (C.immat == 1) {
        d = C.wd[od] + (pval(r.mm[i]) * dt) * drhs[i];
        rr = fabs(d);
      } else {
        // CMMINC (src/cmminc.f90:22-41) on the whole RHS*DTE
        const T x = C.wd[od] + dt * drhs[i], cdt = C.wd[(size_t)C.n_spec_slots * 3 * C.Vp + od];
        d = pval(r.mm[i]) * x + cdt;
        rr = ((x >= (T)0) ? C.cmax[3 * (size_t)e + i] : C.cmin[3 * (size_t)e + i]) * x + cdt;
        rr = rr > (T)0 ? rr : (T)0;
      }
      const T f = fo[o];
      T f1 = f + d;
      const T ch = (f1 < (T)0) ? -f : d;
      f1 = f1 > (T)0 ? f1 : (T)0;
      mx = fmax(mx, (double)rr);
      if (r.flags & (1 << i))
        f1 = C.nfinf[v];
      else
        sq += (double)ch * (double)ch;
      fnw[o] = f1;
    }
  };
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  if (!seq) {
    for (int it = tid; it < C.n_spec_par; it += nt) item(C.spec_par[it]);
  } else {
    for (int s = tid >> 5; s < C.n_spec_slots; s += nt >> 5)
      for (int j0 = C.spec_seq_off[s], j2 = C.spec_seq_off[s + 1]; j0 < j2;) {
        const int j1 = C.spec_seq[2 * j0 + 1];
        for (int j = j0 + (tid & 31); j < j1; j += 32) item(C.spec_seq[2 * j]);
        __syncwarp();
        j0 = j1;
      }
  }
  mx = warp_max(mx);
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0 && (mx > 0.0 || sq > 0.0)) {
    atomicAdd(&C.ctrl->acc_sq, sq);
    atomicMax(reinterpret_cast<unsigned long long*>(&C.ctrl->acc_max), (unsigned long long)__double_as_longlong(mx));
  }
}

// The bookkeeping as a launch of its own, one CTA per case: for sets with
// ALPHA < 1 cases, whose residual is complete after k_wspec.
template <class T> __global__ void k_resid(BatchArgs<T> a) {
  if (threadIdx.x != 0) return;
  const CaseDev<T>& C = a.cases[blockIdx.x];
  if (C.ctrl->done) return;
  resid_book(C, C.ctrl->acc_max, C.ctrl->acc_sq);
}

// ------------------------------------------------- velocity-space shards ----
// A handle that holds only some speed rings of the velocity grid (the
// reference's V-communicator partition, src/spectralbgk.f90:163-199)
// forms partial velocity sums; the caller adds them up over the shards
// between the phases of a step, as the reference's MPI_ALLREDUCEs over
// MPI_COMM_V do (src/macros.f90:114-119, 153-154; src/compmu.f90:80-81;
// src/flucon2.f90:215-216).  Exchange buffers (device, the caller's):
//   sums1 [3][3E]: n, n*ux, n*uy per DG node (MACROS pass 1);
//   sums2 [2][3E] + [nwall]: the pressure sum over M/NA, COMPMU's mean
//          relative-speed sum, FLUCON2's wall sums;
//   res [2]: the step's max residual and sum of squared changes.
// One warp per DG node (a row of f in global memory, 16-byte vectors).
template <class T>
__global__ void __launch_bounds__(256) k_shard_sums1(const __grid_constant__ CaseDev<T> C, double* __restrict__ sums1) {
  if (C.ctrl->done) return;
  const int lane = threadIdx.x & 31, node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (node >= 3 * C.E) return;
  const T* row = C.f[C.ctrl->cur] + (size_t)node * C.Vp;
  double s0 = 0, s1 = 0, s2 = 0;
  RowMath<T>::pass1(row, C.tabs, C.Vp, (int)(C.rowbytes / 16), lane, 32, s0, s1, s2);
  s0 = group_sum<32>(s0);
  s1 = group_sum<32>(s1);
  s2 = group_sum<32>(s2);
  if (lane == 0) {
    const size_t n3 = 3 * (size_t)C.E;
    sums1[node] = s0;
    sums1[n3 + node] = s1;
    sums1[2 * n3 + node] = s2;
  }
}
// the bulk velocity of a node from the summed pass-1 sums (src/macros.f90:126-134)
__device__ __forceinline__ void shard_u(const double* __restrict__ sums1, size_t n3, int node, double& s0,
                                        double& ux, double& uy) {
  s0 = sums1[node];
  ux = uy = 0.0;
  if (s0 >= TINY_D) {
    ux = sums1[n3 + node] / s0;
    uy = sums1[2 * n3 + node] / s0;
  }
}
template <class T>
__global__ void __launch_bounds__(256) k_shard_sums2(const __grid_constant__ CaseDev<T> C,
                                                     const double* __restrict__ sums1, double* __restrict__ sums2) {
  if (C.ctrl->done) return;
  const int lane = threadIdx.x & 31, node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (node >= 3 * C.E) return;
  const size_t n3 = 3 * (size_t)C.E;
  double s0, ux, uy;
  shard_u(sums1, n3, node, s0, ux, uy);
  const T* row = C.f[C.ctrl->cur] + (size_t)node * C.Vp;
  double sp = 0, sc = 0;
  RowMath<T>::pass2(row, C.tabs, C.Vp, (int)(C.rowbytes / 16), lane, 32, ux, uy, sp, sc);
  sp = group_sum<32>(sp);
  sc = group_sum<32>(sc);
  if (lane == 0) {
    sums2[node] = sp;
    sums2[n3 + node] = sc;
  }
}
// FLUCON2's sum over this shard's outgoing velocities, one CTA per wall side
template <class T>
__global__ void __launch_bounds__(WALL_THREADS) k_shard_wall(const __grid_constant__ CaseDev<T> C,
                                                             double* __restrict__ wsum) {
  __shared__ double part[WALL_THREADS / 32];
  if (C.ctrl->done) return;
  const WallSide ws = C.walls[blockIdx.x];
  const T* f = C.f[C.ctrl->cur];
  const T* f1 = f + ((size_t)ws.elem * 3 + ws.in1) * C.Vp;
  const T* f2 = f + ((size_t)ws.elem * 3 + ws.in2) * C.Vp;
  double t = 0;
  for (int v = threadIdx.x; v < C.V; v += WALL_THREADS) {
    const double test = C.cxD[v] * ws.anx + C.cyD[v] * ws.any;
    if (test > 0.0) t += fabs(test) * (0.5 * ((double)f1[v] + (double)f2[v])) * C.wjf[v];
  }
  t = warp_sum(t);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0;
#pragma unroll
    for (int k = 0; k < WALL_THREADS / 32; ++k) u += part[k];
    wsum[blockIdx.x] = u;
  }
}
// the nodes' moments, MU and NFO parameters and the walls' ETA from the
// summed partials
template <class T>
__global__ void __launch_bounds__(256) k_shard_fin(const __grid_constant__ CaseDev<T> C,
                                                   const double* __restrict__ sums1, const double* __restrict__ sums2) {
  if (C.ctrl->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n3 = 3 * (size_t)C.E;
  double mu = 0.0;
  if (t < (int)n3) {
    double s0, ux, uy;
    shard_u(sums1, n3, t, s0, ux, uy);
    mu = node_epilogue(C, t, s0, ux, uy, s0 >= TINY_D ? s0 : 0.0, sums2[t], sums2[n3 + t]);
  }
  if (t < C.nwall) {
    const WallSide ws = C.walls[t];
    const double eta = sums2[2 * n3 + t] / ws.sumbottom;
    C.bEtaD[ws.bside] = eta;
    C.bwall[4 * (size_t)ws.bside + 3] = (T)((double)C.alpha * eta);
  }
  const double m = warp_max(mu);
  if ((threadIdx.x & 31) == 0 && m > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(&C.ctrl->maxmu), (unsigned long long)__double_as_longlong(m));
}
// the step's residual partials out; after the sum / max over the shards,
// the bookkeeping of k_resid with the global values
template <class T> __global__ void k_shard_respart(const __grid_constant__ CaseDev<T> C, double* __restrict__ res) {
  if (threadIdx.x != 0 || C.ctrl->done) return;
  res[0] = C.ctrl->acc_max;
  res[1] = C.ctrl->acc_sq;
}
template <class T>
__global__ void k_shard_resid(const __grid_constant__ CaseDev<T> C, const double* __restrict__ res) {
  if (threadIdx.x != 0) return;
  if (C.ctrl->done) return;
  resid_book(C, res[0], res[1]);
}

// -------------------------------------------------------------- nodal ----
// MACROS tail (src/macros.f90:156-188) and GETMAC with one partition.
struct NodalArgs {
  const int* node_off;
  const int* node_dg;
  const double* node_ae;
  const double* nraw;
  const double* disux;
  const double* disuy;
  const double* disps;
  double *nd, *rho, *u, *v, *ps, *temp;
  int NP;
  double MM, R;
};

// mesh node q's ND, RHO, UVEL, VVEL, PS, TEMP into out[k*stride + q]
__device__ __forceinline__ void nodal_one(const NodalArgs& a, int q, double* out, int stride) {
  double flag = 0, nd = 0, u = 0, v = 0, ps = 0;
  for (int k = a.node_off[q]; k < a.node_off[q + 1]; ++k) {
    const int dg = a.node_dg[k];
    const double ae = a.node_ae[k];
    flag += ae;
    nd += a.nraw[dg] * ae;
    if (a.nraw[dg] >= TINY_D) {
      u += ae * a.disux[dg];
      v += ae * a.disuy[dg];
    }
    ps += a.disps[dg] * ae;
  }
  double rho = 0, t = 0;
  if (nd < TINY_D) {
    u = v = ps = 0;
  } else {
    nd = nd / flag;
    rho = nd * a.MM;
    u = u / flag;
    v = v / flag;
    ps = ps / flag;
    t = ps / (a.R * rho);
  }
  out[q] = nd;
  out[stride + q] = rho;
  out[2 * stride + q] = u;
  out[3 * stride + q] = v;
  out[4 * stride + q] = ps;
  out[5 * stride + q] = t;
}

__global__ void k_nodal(NodalArgs a) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.NP) return;
  nodal_one(a, q, a.nd, (int)(a.rho - a.nd));
}

// ------------------------------------------------ observables on device ----
// GETMAC's nodal fields and GETFOR's lift and drag (src/getmac.f90:98-123,
// src/getfor.f90:29-49) recorded without a host round trip.  A record is
// [ITIME, LIFT, DRAG, 0][ND | RHO | UVEL | VVEL | PS | TEMP] (6*NPOIN).
// Ring mode (inside the step graph, right after the moment kernel, whose
// moments are those of the state after the previous step): the record of
// ITIME = itime0 + step is taken when that is a multiple of `every`, into
// slot count % cap of the ring, and count is bumped.  Direct mode
// (force_itime >= 0): one record into `direct`, unconditionally.
struct OutArgs {
  NodalArgs nod;  // its nd .. temp pointers unused
  const Ctrl* ctrl;
  const ForceSide* fs;
  int nfs;
  int every, cap;
  double* ring;   // [cap][4 + 6*NP]
  int* count;
  double* direct;
  int force_itime;
};
__device__ __forceinline__ int out_itime(const OutArgs& o) {
  if (o.force_itime >= 0) return o.force_itime;
  const Ctrl* c = o.ctrl;
  if (c->done || c->step == 0) return -1;
  const int it = c->itime0 + c->step;
  return (it % o.every == 0) ? it : -1;
}
__device__ __forceinline__ double* out_record(const OutArgs& o) {
  if (o.direct) return o.direct;
  return o.ring + (size_t)(*o.count % o.cap) * (4 + 6 * (size_t)o.nod.NP);
}
__global__ void k_out_nodal(OutArgs o) {
  if (out_itime(o) < 0) return;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= o.nod.NP) return;
  nodal_one(o.nod, q, out_record(o) + 4, o.nod.NP);
}
constexpr int FORCE_THREADS = 256;
__global__ void __launch_bounds__(FORCE_THREADS) k_out_forces(OutArgs o) {
  const int it = out_itime(o);
  if (it < 0) return;
  double* rec = out_record(o);
  const double* ps = rec + 4 + 4 * (size_t)o.nod.NP;
  double lift = 0.0, drag = 0.0;
  for (int k = threadIdx.x; k < o.nfs; k += FORCE_THREADS) {
    const ForceSide s = o.fs[k];
    const double pav = 0.5 * (ps[s.ip1] + ps[s.ip2]);
    lift -= pav * s.ly;
    drag -= pav * s.lx;
  }
  __shared__ double red[2][FORCE_THREADS / 32];
  lift = warp_sum(lift);
  drag = warp_sum(drag);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = lift;
    red[1][threadIdx.x >> 5] = drag;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double l = 0.0, d = 0.0;
    for (int w = 0; w < FORCE_THREADS / 32; ++w) {
      l += red[0][w];
      d += red[1][w];
    }
    rec[0] = (double)it;
    rec[1] = l;
    rec[2] = d;
    rec[3] = 0.0;
    if (!o.direct) {
      __threadfence();
      *o.count += 1;
    }
  }
}

// ---------------------------------------------- vector extrapolation ----
// Reduced-rank extrapolation of the pseudo-time iterates (no counterpart in
// the reference; it changes the path to the fixed point, not the fixed
// point): snapshots x_0 .. x_{n-1} of the state, differences
// u_j = x_{j+1} - x_j.  k_gram accumulates G_ab = u_a . u_b (a <= b < n-1)
// in FP64 (per-thread partials, a warp and block reduction, one atomic per
// block and entry); k_combine writes max(sum_j gamma_j x_j, 0).
//
// k_gram reads the snapshots once, a 16-byte vector of each in flight per
// thread, and is compiled for every number m of differences, so that a small
// m does not carry the sums of ten.  With 8-byte loads and all 55 sums it ran
// at 1.9 TB/s (322 us for ten snapshots of 61 MB).
constexpr int RRE_MAX = 11;  // snapshots (10 differences, 55 products)
template <class T, int M>
__global__ void __launch_bounds__(256) k_gram(const T* __restrict__ snaps, size_t stride, size_t N,
                                              double* __restrict__ G) {
  constexpr int NPAIR = M * (M + 1) / 2, W = 16 / (int)sizeof(T);
  using V = typename Pair<T>::vec;
  double acc[NPAIR];
#pragma unroll
  for (int q = 0; q < NPAIR; ++q) acc[q] = 0.0;
  // N is a multiple of W (the rows' pitch is one of 32)
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N / W; i += (size_t)gridDim.x * blockDim.x) {
    V x[M + 1];
#pragma unroll
    for (int j = 0; j <= M; ++j) x[j] = __ldg(reinterpret_cast<const V*>(snaps + (size_t)j * stride) + i);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      double u[M];
#pragma unroll
      for (int j = 0; j < M; ++j) u[j] = (double)vec_at(x[j + 1], w) - (double)vec_at(x[j], w);
#pragma unroll
      for (int a = 0, q = 0; a < M; ++a)
#pragma unroll
        for (int b = a; b < M; ++b, ++q) acc[q] = fma(u[a], u[b], acc[q]);
    }
  }
  __shared__ double red[8][NPAIR];
#pragma unroll
  for (int q = 0; q < NPAIR; ++q) {
    const double v = warp_sum(acc[q]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = v;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < NPAIR; q += blockDim.x) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w][q];
    int a = 0, o = q;
    while (o >= M - a) o -= M - a++;
    atomicAdd(&G[a * M + a + o], t);
  }
}

template <class T>
__global__ void __launch_bounds__(256) k_combine(const T* __restrict__ snaps, size_t stride, int m,
                                                 const double* __restrict__ gamma, size_t N, T* __restrict__ out) {
  __shared__ double g[RRE_MAX];
  if (threadIdx.x < RRE_MAX) g[threadIdx.x] = (int)threadIdx.x < m ? gamma[threadIdx.x] : 0.0;
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
    double x = 0.0;
    for (int j = 0; j < m; ++j) x = fma(g[j], (double)snaps[(size_t)j * stride + i], x);
    out[i] = (T)(x > 0.0 ? x : 0.0);
  }
}

// ----------------------------------------------------- layout changes ----
// reference DISNF(3,V,E) (old element order) <-> f rows (plan order, pitch Vp)
template <class S, class T>
__global__ void k_to_internal(const S* __restrict__ src, T* __restrict__ dst, const int* __restrict__ inv, int V,
                              int Vp) {
  const int eo = blockIdx.x;
  const size_t en = (size_t)inv[eo];
  const S* s = src + (size_t)eo * 3 * V;
  for (int i = 0; i < 3; ++i)
    for (int v = threadIdx.x; v < V; v += blockDim.x) dst[(en * 3 + i) * Vp + v] = (T)s[(size_t)v * 3 + i];
}

template <class T, class S>
__global__ void k_from_internal(const T* __restrict__ src, S* __restrict__ dst, const int* __restrict__ inv, int V,
                                int Vp) {
  const int eo = blockIdx.x;
  const size_t en = (size_t)inv[eo];
  S* d = dst + (size_t)eo * 3 * V;
  for (int i = 0; i < 3; ++i)
    for (int v = threadIdx.x; v < V; v += blockDim.x) d[(size_t)v * 3 + i] = (S)src[(en * 3 + i) * Vp + v];
}

// INICON2 (src/inicon2.f90:143-174) times an optional per-DG-node scale.
template <class T>
__global__ void k_init_uniform(T* __restrict__ f, const double* __restrict__ g, const double* __restrict__ scale,
                               double n1, int V, int Vp, size_t ndg) {
  const size_t dg = blockIdx.x;
  if (dg >= ndg) return;
  const double sc = scale ? scale[dg] : 1.0;
  for (int v = threadIdx.x; v < V; v += blockDim.x) {
    double val = n1 * g[v];
    if (scale) val = val * sc;
    f[dg * Vp + v] = (T)val;
  }
}

// Maxwellian from per-DG-node (n, u, v, T) (the warm start): the INICON2
// formula with RHO = n*M/NA, P = RHO*R*T, BETA^2 = RHO/(2P).
template <class T>
__global__ void k_init_maxwellian(T* __restrict__ f, const double* __restrict__ prm /* [dg][4] */,
                                  const double* __restrict__ cx, const double* __restrict__ cy, double MM,
                                  double R, int V, int Vp, size_t ndg) {
  const size_t dg = blockIdx.x;
  if (dg >= ndg) return;
  const double n = prm[4 * dg], u = prm[4 * dg + 1], w = prm[4 * dg + 2], t = prm[4 * dg + 3];
  const bool live = n >= TINY_D && t > 0.0;
  const double rho = n * MM, p = rho * R * t;
  const double b2 = live ? rho / (2 * p) : 0.0;
  for (int v = threadIdx.x; v < V; v += blockDim.x) {
    double val = 0.0;
    if (live) {
      const double dx = cx[v] - u, dy = cy[v] - w;
      val = n * ((b2 / PI_D) * exp(-(b2 * (dx * dx + dy * dy))));
    }
    f[dg * Vp + v] = (T)val;
  }
}

}  // namespace dgbgk
