// FP64 PCG of POT3D on sm_100a: matrix-free 7-point spherical stencil,
// diagonal preconditioner, fused dot/axpy reductions, boundary and periodic
// phi seam handled inline, and the potfld pieces around the solve (RHS by
// the boundary trick, phi finalisation, getb + magnetic energy).
//
// Per PCG iteration (classical PCG of cgsolve, src/pot3d.F90:4336-4365)
// two kernels run, both tiled over (i, j, k) with TIxTJ tiles that march
// along k:
//   k_stencil<PCG> : p = beta*p + z (z = a_i*r formed on the fly),
//                    q = A p, and the p.q partial sums -> alpha
//   k_update<>     : x += alpha p, r -= alpha q, z = a_i*r, r.z -> rho,
//                    beta, epsn (ernorm, src/pot3d.F90:4430-4433); on grids
//                    above L2 x is left to k_update_x_group, once a group
// All scalars stay on the device (SolveState); the host only polls the
// convergence flag between CUDA-graph launches of several iterations.
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "pot3d_internal.cuh"
#include "pot3d_solver.h"
#include "tma.cuh"

using namespace pot3d;

static thread_local std::string g_last_error;
void pot3d_set_error(const std::string &msg) { g_last_error = msg; }
int pot3d_cuda_status(cudaError_t e, const char *where) {
  if (e == cudaSuccess) return POT3D_OK;
  pot3d_set_error(std::string(where) + ": " + cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? POT3D_ERR_NOMEM : POT3D_ERR_CUDA;
}
extern "C" const char *pot3d_gpu_last_error(void) { return g_last_error.c_str(); }


// ============================================================================
// Stencil coefficients (load_matrix_pot3d_solve, src/pot3d.F90:4590-4611).
// Each coefficient is formed with the same operand order as the reference so
// the values are bit-identical; __dmul_rn/__dadd_rn keep the compiler from
// contracting them into FMAs.
// ============================================================================
struct RowCoef {  // per theta row j
  double sd;      // sth(j)*dth(j)
  double stm, dtim, stp, dtip;
};
struct PtCoef {   // per radial point i in row j
  double c17;     // (drh(i)*dth(j))*sth_i(j)
  double drh, r2m, drim, r2p, drip;
};
struct Coef7 {
  double a1, a2, a3, a4, a5, a6, a7;
};

__device__ __forceinline__ RowCoef row_coef(const DevMesh &m, int j) {
  RowCoef c;
  c.sd = __dmul_rn(m.sth[j], m.dth[j]);
  c.stm = m.st[j - 1];
  c.dtim = m.dt_i[j - 1];
  c.stp = m.st[j];
  c.dtip = m.dt_i[j];
  return c;
}
__device__ __forceinline__ PtCoef pt_coef(const DevMesh &m, int i, int j) {
  PtCoef c;
  c.drh = m.drh[i];
  c.c17 = __dmul_rn(__dmul_rn(c.drh, m.dth[j]), m.sth_i[j]);
  c.r2m = m.r2[i - 1];
  c.drim = m.dr_i[i - 1];
  c.r2p = m.r2[i];
  c.drip = m.dr_i[i];
  return c;
}
__device__ __forceinline__ Coef7 coef7(const PtCoef &p, const RowCoef &r, double dpim, double dpip,
                                       double dphk) {
  Coef7 a;
  a.a1 = -__dmul_rn(p.c17, dpim);
  a.a7 = -__dmul_rn(p.c17, dpip);
  const double u = __dmul_rn(p.drh, dphk);
  a.a2 = -__dmul_rn(__dmul_rn(u, r.stm), r.dtim);
  a.a6 = -__dmul_rn(__dmul_rn(u, r.stp), r.dtip);
  const double v = __dmul_rn(r.sd, dphk);
  a.a3 = -__dmul_rn(__dmul_rn(v, p.r2m), p.drim);
  a.a5 = -__dmul_rn(__dmul_rn(v, p.r2p), p.drip);
  a.a4 = -__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(a.a1, a.a2), a.a3), a.a5), a.a6), a.a7);
  return a;
}
// delsq's sum, src/pot3d.F90:5364-5372, in the reference's term order.
__device__ __forceinline__ double apply7(const Coef7 &a, double xkm, double xjm, double xim, double xc,
                                         double xip, double xjp, double xkp) {
  double y = a.a1 * xkm;
  y = fma(a.a2, xjm, y);
  y = fma(a.a3, xim, y);
  y = fma(a.a4, xc, y);
  y = fma(a.a5, xip, y);
  y = fma(a.a6, xjp, y);
  y = fma(a.a7, xkp, y);
  return y;
}

// The stencil kernels use the coefficients in factored form: with
//   g1 = drh*dth*sth_i, g2 = drh*st(j-1)*dt_i(j-1), g6 = drh*st(j)*dt_i(j),
//   g3 = sth*dth*r2(i-1)*dr_i(i-1), g5 = sth*dth*r2(i)*dr_i(i)
// the seven coefficients of load_matrix_pot3d_solve are
//   a1 = -g1*dp_i(k-1), a7 = -g1*dp_i(k), a2 = -g2*dph(k), a6 = -g6*dph(k),
//   a3 = -g3*dph(k), a5 = -g5*dph(k), a4 = -(a1+a2+a3+a5+a6+a7),
// so y = a4*x - g1*(dp_i(k-1)*x(k-1) + dp_i(k)*x(k+1))
//          - dph(k)*(g2*x(j-1) + g3*x(i-1) + g5*x(i+1) + g6*x(j+1)).
// This evaluates the same operator with short dependency chains; values
// differ from the stored-coefficient form by rounding only.
struct PtFac {
  double g1, g2, g3, g5, g6, gs;  // gs = g2+g3+g5+g6
};
__device__ __forceinline__ PtFac pt_fac(const DevMesh &m, int i, int j) {
  PtFac f;
  const double drh = m.drh[i];
  const double sd = m.sth[j] * m.dth[j];
  f.g1 = drh * m.dth[j] * m.sth_i[j];
  f.g2 = drh * m.st[j - 1] * m.dt_i[j - 1];
  f.g6 = drh * m.st[j] * m.dt_i[j];
  f.g3 = sd * m.r2[i - 1] * m.dr_i[i - 1];
  f.g5 = sd * m.r2[i] * m.dr_i[i];
  f.gs = (f.g2 + f.g6) + (f.g3 + f.g5);
  return f;
}
__device__ __forceinline__ double apply_fac(const PtFac &f, double dpim, double dpip, double dphk, double xkm,
                                            double xjm, double xim, double xc, double xip, double xjp, double xkp) {
  const double a4 = fma(f.g1, dpim + dpip, f.gs * dphk);
  const double tk = fma(dpim, xkm, dpip * xkp);
  const double tr = fma(f.g3, xim, f.g5 * xip);
  const double tt = fma(f.g2, xjm, f.g6 * xjp);
  const double off = fma(f.g1, tk, dphk * (tr + tt));
  return fma(a4, xc, -off);
}

// ============================================================================
// Stencil kernel.  MODE_AX: y = A x (ax, src/pot3d.F90:5102-5150) with the
// south-pole ring sums S1 supplied.  MODE_PCG: p_new = beta*p + a_i*r on the
// fly, q = A p_new, p_new.q.  MODE_PCGZ: same with z read from an FP32
// vector (the ILU(0) preconditioner's output).  MODE_PCG32 / MODE_PCGZ32:
// the FP32-inner forms of PCG / PCGZ: p, r, z and q are stored in FP32 and
// read as FP32 boxes; p_new is rounded once, and A p_new is evaluated in FP64
// registers, so q is the FP64 product of the stored FP32 p_new rounded once.  (An FP32 evaluation of a4*x - sum(a_nb*x_nb)
// cancels away the smooth modes that set the convergence of this
// operator; FP64 arithmetic costs nothing here, the kernel is HBM-bound.)
//
// Boundaries (set_boundary_points with vmask=0, src/pot3d.F90:5413-5484):
//   i=1  ghost = x(2)            (r0 Neumann)
//   i=nr ghost = pm_r1 * x(nrm1)
//   j=1  ghost enters through a2 = -drh*dph*st(1)*dt_i(1) = 0 (st(1)=sin 0)
//   j=nt ghost = 2*S1(i) - x(i,ntm1,k), S1 the ring mean of x at j=ntm1
//   k    periodic wrap (seam_hhh, src/pot3d.F90:5746-5758)
//
// A thread marches along k with its own column's three planes in registers
// and reads only the neighbours in e and j from shared memory, two columns per
// access.  Measured against every neighbour read from the ring: PCGZ32 53.8 ->
// 49.9 us at 127x181x361 (344 -> 315 at 255x361x721); whole solves, 127x181x361
// FP32-refined diagonal 336 -> 302 ms and 121x181x361 FP64 diagonal 506 -> 455
// to 475 ms.
// ============================================================================
enum { MODE_AX = 0, MODE_PCG = 1, MODE_PCGZ = 2, MODE_PCG32 = 3, MODE_PCGZ32 = 4 };

struct StencilArgs {
  const double *x;          // AX input
  double *y;                // AX output
  const double *p_old;      // PCG
  const double *r;          // PCG
  const float *ai;          // PCG diagonal preconditioner
  const float *z32;         // PCGZ
  double *p_new;            // PCG out
  double *q;                // PCG out
  const float *p_old32;     // PCG32: FP32 inner vectors
  const float *r32;
  float *p_new32;
  float *q32;
  const double *s1_direct;  // AX: S1(e), length NRP
  const double *s1z_part;   // PCG: [nkc][NRP] ring partial sums of z
  double *s1p;              // PCG: [2][NRP] ring sums of p (parity buffers)
  SolveState *st;
  double *partials;
  int xslot1;               // 1 + the slot of st->xa that receives alpha (0: none)
};

// Shared-memory layout of the TMA-staged stencil.  Each pipeline stage holds
// one k-plane of the tile plus a one-point halo: FP64 boxes of 68 x 10
// points starting at (i = ib-2, j = j0-1) and FP32 boxes of 72 x 10 starting
// at (i = ib-4, j = j0-1), so every TMA x-coordinate is 16-byte aligned.
// Rows or columns outside the vector are zero-filled by the TMA unit; the
// physical ghosts are applied when the stencil is evaluated.
constexpr int S_STAGES = 4;
constexpr int BOX_Y = TJ + 2;
constexpr int BOX64_X = TI + 4;
constexpr int BOX32_X = TI + 8;
constexpr int TILE64_BYTES = BOX64_X * BOX_Y * 8;
constexpr int TILE32_BYTES = BOX32_X * BOX_Y * 4;
constexpr int TILE64_PITCH = (TILE64_BYTES + 127) / 128 * 128;
constexpr int TILE32_PITCH = (TILE32_BYTES + 127) / 128 * 128;
constexpr int PN_SLOTS = 3;  // p_new planes in the ring: written, read, and still read by slower warps
constexpr int MAX_TK = 512;  // k-planes per block at most (per-k factors in shared memory)
constexpr uint32_t WAIT_LIMIT = 1u << 24;

template <int MODE>
struct StageCfg;
template <>
struct StageCfg<MODE_AX> {
  static constexpr int n64 = 1, n32 = 0;
};
template <>
struct StageCfg<MODE_PCG> {
  static constexpr int n64 = 2, n32 = 1;
};
template <>
struct StageCfg<MODE_PCGZ> {
  static constexpr int n64 = 1, n32 = 1;
};
template <>
struct StageCfg<MODE_PCG32> {
  static constexpr int n64 = 0, n32 = 3;
};
template <>
struct StageCfg<MODE_PCGZ32> {
  static constexpr int n64 = 0, n32 = 2;
};
template <int MODE>
struct StageLayout {
  static constexpr int n64 = StageCfg<MODE>::n64, n32 = StageCfg<MODE>::n32;
  static constexpr int bytes = n64 * TILE64_PITCH + n32 * TILE32_PITCH;
  static constexpr uint32_t tx = n64 * TILE64_BYTES + n32 * TILE32_BYTES;
  static constexpr int kfac_off = S_STAGES * bytes + PN_SLOTS * TILE64_BYTES + 128;
  static constexpr int smem = kfac_off + 4 * 8 * MAX_TK;
};

// Tensor maps of the stage inputs: m64[0] = x | p_old, m64[1] = r, m32 = a_i | z;
// FP32 modes: m32[0] = p_old, m32[1] = r (PCG32) | z (PCGZ32), m32[2] = a_i (PCG32).
struct StencilMaps {
  CUtensorMap m64[2];
  CUtensorMap m32[3];
};

template <typename T>
struct Vec2;
template <>
struct Vec2<double> {
  using type = double2;
};
template <>
struct Vec2<float> {
  using type = float2;
};

template <typename T2>
__device__ __forceinline__ double2 widen2(const T2 v) {
  return make_double2((double)v.x, (double)v.y);
}

template <int MODE>
__device__ __forceinline__ void stencil_body(const StencilMaps &maps, const Geo &g, const DevMesh &m,
                                             const StencilArgs &a, const int bx, const int by, const int bz) {
  using L = StageLayout<MODE>;
  constexpr bool F32 = MODE == MODE_PCG32 || MODE == MODE_PCGZ32;
  using T = typename std::conditional<F32, float, double>::type;  // storage of p_new and q
  using T2 = typename Vec2<T>::type;
  extern __shared__ __align__(1024) unsigned char dyn[];
  __shared__ __align__(8) uint64_t bar[S_STAGES];
  __shared__ double red[NTHR / 32];
  __shared__ double s1sh[TI];
  __shared__ int abort_flag;

  double *kfac = reinterpret_cast<double *>(dyn + L::kfac_off);  // [tk][4]: dp_i(k-1), dp_i(k), dph(k)
  unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 127) & ~uintptr_t(127));
  // p_new ring [PN_SLOTS][BOX_Y][BOX64_X], FP64 in every mode: the FP32 modes
  // store each rounded p_new widened once, so the stencil reads it without
  // a conversion per neighbour (conversions issue at a fraction of the FP64
  // rate)
  double *pn_ring = reinterpret_cast<double *>(base + S_STAGES * L::bytes);

  const int tid = threadIdx.x;
  const int lane = tid & 31, w = tid >> 5;
  const int ib = bx * TI;
  const int el = 2 * lane;
  const int e0 = ib + el;
  const int j0 = by * TJ;
  const int jj = j0 + w;
  const int k0 = bz * g.tk;
  const int k1 = min(k0 + g.tk, g.npm2);
  const bool rowv = jj < g.ntm2;
  const bool v0 = rowv && e0 < g.nrm2;
  const bool v1 = rowv && e0 + 1 < g.nrm2;
  const bool south = rowv && jj == g.ntm2 - 1;

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < S_STAGES; s++) mbar_init(&bar[s], 1);
    mbar_init_fence();
    if (L::n64 > 0) tma_prefetch_desc(&maps.m64[0]);
    if (L::n64 > 1) tma_prefetch_desc(&maps.m64[1]);
    for (int q = 0; q < L::n32; q++) tma_prefetch_desc(&maps.m32[q]);
  }
  if (tid < TI) s1sh[tid] = 0.0;
  PtFac f0, f1;
  auto mesh_factors = [&]() {
    const int jf = jj + 2;
    if (rowv) {
      f0 = pt_fac(m, min(e0, g.nrm2 - 1) + 2, jf);
      f1 = pt_fac(m, min(e0 + 1, g.nrm2 - 1) + 2, jf);
    }
    // dp_i(k-1), dp_i(k), dph(k) of the block's planes, staged once.
    for (int q = tid; q < k1 - k0; q += NTHR) {
      const int kf = k0 + q + 2;
      kfac[4 * q + 0] = m.dp_i[kf - 1];
      kfac[4 * q + 1] = m.dp_i[kf];
      kfac[4 * q + 2] = m.dph[kf];
    }
  };
  // The diagonal modes are launched before the kernel they follow has ended
  // and form the mesh factors meanwhile; the others form them behind the
  // first loads.
  constexpr bool EARLY = MODE == MODE_PCG || MODE == MODE_PCG32;
  if constexpr (EARLY) {
    mesh_factors();
    pdl_wait();
    pdl_trigger();
  }
  double beta = 0.0;
  int par = 0;
  if (MODE != MODE_AX) {
    const volatile SolveState *vs = a.st;
    if (vs->status != ST_RUNNING) {  // uniform: converged or failed
      // no iteration: the grouped x update applies nothing for it
      if (a.xslot1 && bx == 0 && by == 0 && bz == 0 && threadIdx.x == 0) a.st->xa[a.xslot1 - 1] = 0.0;
      return;
    }
    beta = vs->beta;
    par = vs->par;
  }
  __syncthreads();

  const int p_first = k0 - 1;         // planes p_first .. k1 feed the stencil
  const int n_planes = k1 - k0 + 2;
  int kk_issue = k0 == 0 ? g.npm2 - 1 : k0 - 1;  // plane of the next issue (periodic)
  auto issue = [&](int local) {       // thread 0: TMA loads of one plane
    const int kk = kk_issue;
    kk_issue = kk + 1 == g.npm2 ? 0 : kk + 1;
    const int s = local % S_STAGES;
    unsigned char *st = base + s * L::bytes;
    mbar_expect_tx(&bar[s], L::tx);
    for (int q = 0; q < L::n64; q++) tma_load_3d(st + q * TILE64_PITCH, &maps.m64[q], ib - 2, j0 - 1, kk, &bar[s]);
    for (int q = 0; q < L::n32; q++)
      tma_load_3d(st + L::n64 * TILE64_PITCH + q * TILE32_PITCH, &maps.m32[q], ib - 4, j0 - 1, kk, &bar[s]);
  };
  int issued = 0;
  if (tid == 0) {
    for (; issued < S_STAGES && issued < n_planes; issued++) issue(issued);
  }

  // South-pole ring sums for the tile's radial points (last theta row only).
  if (MODE == MODE_AX) {
    if (tid < TI && ib + tid < g.nrm2) s1sh[tid] = a.s1_direct[ib + tid];
  } else if (j0 + TJ >= g.ntm2) {
    // S1(p_new) = beta*S1(p_old) + S1(z): the ring sums are linear in p.
    if (tid < TI && ib + tid < g.nrm2) {
      const int e = ib + tid;
      double sz = 0.0;
      for (int c = 0; c < g.nkc_u; c++) sz += a.s1z_part[(long long)c * g.NRP + e];
      const double s = fma(beta, a.s1p[par * g.NRP + e], sz);
      s1sh[tid] = s;
      if (bz == 0) a.s1p[(par ^ 1) * g.NRP + e] = s;
    }
  }

  if constexpr (!EARLY) mesh_factors();
  __syncthreads();
  const double s1a = south ? s1sh[el] : 0.0, s1b = south ? s1sh[el + 1] : 0.0;
  const double pm = m.pm_r1;
  double dot = 0.0;

  // p_new of two neighbouring columns (col even) or of one at (row, col) of
  // the stage tile; col counts FP64 columns.  PCG32 forms p_new in FP64 and
  // rounds it once: an FP32 pair (exact products, an exact sum) in its place is
  // 2% faster but up to 30 times further off under cancellation, and 14% slower
  // with a test of its rounding (302, 297 and 343 ms a solve at 127x181x361).
  // PCGZ32 forms p_new with one FP32 fma (beta rounded to FP32 once per block):
  // every operand is already FP32 and the result is stored in FP32.
  const float beta32 = (float)beta;
  auto p64 = [&](float pv, float ai, float r) -> float {
    return (float)fma(beta, (double)pv, (double)ai * (double)r);
  };
  auto pnew_at = [&](const unsigned char *st, int row, int col, auto pair) {
    constexpr bool PAIR = decltype(pair)::value;
    using D = typename std::conditional<PAIR, double2, double>::type;
    using F = typename std::conditional<PAIR, float2, float>::type;
    const int c64 = row * BOX64_X + col, c32 = row * BOX32_X + col + 2;
    auto f32 = [&](int q) { return *reinterpret_cast<const F *>(reinterpret_cast<const float *>(st + q) + c32); };
    auto f64 = [&](int q) { return *reinterpret_cast<const D *>(reinterpret_cast<const double *>(st + q) + c64); };
    if constexpr (MODE == MODE_AX) {
      return f64(0);
    } else if constexpr (MODE == MODE_PCG32) {
      const F pv = f32(0), r = f32(TILE32_PITCH), ai = f32(2 * TILE32_PITCH);
      if constexpr (PAIR)
        return make_float2(p64(pv.x, ai.x, r.x), p64(pv.y, ai.y, r.y));
      else
        return p64(pv, ai, r);
    } else if constexpr (MODE == MODE_PCGZ32) {
      const F pv = f32(0), z = f32(TILE32_PITCH);
      if constexpr (PAIR)
        return make_float2(__fmaf_rn(beta32, pv.x, z.x), __fmaf_rn(beta32, pv.y, z.y));
      else
        return __fmaf_rn(beta32, pv, z);
    } else if constexpr (MODE == MODE_PCG) {
      const D pv = f64(0), r = f64(TILE64_PITCH);
      const F ai = f32(2 * TILE64_PITCH);
      if constexpr (PAIR)
        return make_double2(fma(beta, pv.x, (double)ai.x * r.x), fma(beta, pv.y, (double)ai.y * r.y));
      else
        return fma(beta, pv, (double)ai * r);
    } else {
      const D pv = f64(0);
      const F z = f32(TILE64_PITCH);
      if constexpr (PAIR)
        return make_double2(fma(beta, pv.x, (double)z.x), fma(beta, pv.y, (double)z.y));
      else
        return fma(beta, pv, (double)z);
    }
  };

  // A thread's own column stays in registers (x at planes k-1, k, k+1); the
  // ring serves the neighbours in e and j only.
  T2 own_cur{}, own_prev{};
  double2 xm{}, xc{}, xn{};
  const int own = (w + 1) * BOX64_X + 2 + el;
  const bool first_e = e0 == 0, last_e0 = e0 == g.nrm2 - 1, last_e1 = e0 + 1 == g.nrm2 - 1;
  long long id = g.idx(e0, jj, k0);
  const long long id_step = (long long)g.NRP * g.ntm2;
  double *slot = pn_ring;             // plane `local`
  double *const ring_end = pn_ring + PN_SLOTS * (BOX_Y * BOX64_X);
  int local = 0;
  for (; local < n_planes; local++) {
    const int s = local % S_STAGES;
    const uint32_t parity = (local / S_STAGES) & 1;
    if (!mbar_wait(&bar[s], parity, WAIT_LIMIT)) abort_flag = 1;
    const unsigned char *st = base + s * L::bytes;
    // own pair (kept in registers in storage precision for the output of
    // this plane, which follows one plane later)
    own_prev = own_cur;
    own_cur = pnew_at(st, w + 1, 2 + el, std::true_type{});
    xm = xc;
    xc = xn;
    xn = make_double2((double)own_cur.x, (double)own_cur.y);
    *reinterpret_cast<double2 *>(slot + own) = xn;
    {  // halo: theta rows 0 and TJ+1 (128 points) and radial columns (16)
      if (tid < 2 * TI) {
        const int row = (tid < TI) ? 0 : TJ + 1;
        const int col = 2 + (tid & (TI - 1));
        slot[row * BOX64_X + col] = (double)pnew_at(st, row, col, std::false_type{});
      } else if (tid < 2 * TI + 2 * TJ) {
        const int q = tid - 2 * TI;
        const int row = 1 + (q >> 1);
        const int col = (q & 1) ? TI + 2 : 1;
        slot[row * BOX64_X + col] = (double)pnew_at(st, row, col, std::false_type{});
      }
    }
    __syncthreads();
    if (abort_flag) break;
    if (tid == 0 && issued < n_planes) {  // refill the stage just consumed
      issue(issued);
      issued++;
    }
    const double *sc = slot == pn_ring ? ring_end - BOX_Y * BOX64_X : slot - BOX_Y * BOX64_X;  // plane local - 1
    slot = slot + BOX_Y * BOX64_X == ring_end ? pn_ring : slot + BOX_Y * BOX64_X;
    if (local >= 2 && v0) {  // the stencil of plane kq = local - 2 of the chunk is complete
      const double *kf = kfac + 4 * (local - 2);
      const double2 dpi = *reinterpret_cast<const double2 *>(kf);
      const double dpim = dpi.x, dpip = dpi.y, dphk = kf[2];
      const double2 xjm2 = *reinterpret_cast<const double2 *>(sc + own - BOX64_X);
      double2 xjp2 = *reinterpret_cast<const double2 *>(sc + own + BOX64_X);
      const double xl = sc[own - 1], xr = sc[own + 2];
      // j = 1: the coupling to the row below is an exact zero (st(1) = 0), and
      // the row read there is zero
      if (south) xjp2 = make_double2(2.0 * s1a - xc.x, 2.0 * s1b - xc.y);
      const double xim = first_e ? xc.x : xl;
      const double xip = last_e0 ? pm * xc.x : xc.y;
      const double y = apply_fac(f0, dpim, dpip, dphk, xm.x, xjm2.x, xim, xc.x, xip, xjp2.x, xn.x);
      double y1 = 0.0;
      if (v1) {
        const double xip1 = last_e1 ? pm * xc.y : xr;
        y1 = apply_fac(f1, dpim, dpip, dphk, xm.y, xjm2.y, xc.x, xc.y, xip1, xjp2.y, xn.y);
      }
      if constexpr (MODE == MODE_AX) {
        *reinterpret_cast<double2 *>(a.y + id) = make_double2(y, y1);
      } else if constexpr (F32) {
        // q is stored rounded; p.q uses the stored values, as the update does
        // (own_prev is the stored p_new of this plane; xc holds it exactly)
        const float2 qv = make_float2((float)y, (float)y1);
        const float2 own2 = make_float2(own_prev.x, v1 ? own_prev.y : 0.0f);
        *reinterpret_cast<float2 *>(a.q32 + id) = qv;
        *reinterpret_cast<float2 *>(a.p_new32 + id) = own2;
        dot = fma(xc.x, (double)qv.x, dot);
        dot = fma(v1 ? xc.y : 0.0, (double)qv.y, dot);
      } else {
        const double2 own2 = make_double2(xc.x, v1 ? xc.y : 0.0);
        *reinterpret_cast<double2 *>(a.q + id) = make_double2(y, y1);
        *reinterpret_cast<double2 *>(a.p_new + id) = own2;
        dot = fma(own2.x, y, dot);
        dot = fma(own2.y, y1, dot);
      }
      id += id_step;
    }
  }

  if (abort_flag) {
    // Drain the loads still in flight (bounded), report, and leave.
    if (tid == 0) {
      for (int l = local; l < issued; l++) mbar_wait(&bar[l % S_STAGES], (l / S_STAGES) & 1, WAIT_LIMIT);
      if (MODE != MODE_AX) {
        // no block is the last to arrive now, so nothing else writes the slot,
        // which still holds an earlier group's alpha
        if (a.xslot1) a.st->xa[a.xslot1 - 1] = 0.0;
        atomicExch(&a.st->status, ST_TIMEOUT);
      }
    }
    return;
  }
  if (MODE != MODE_AX) {
    double bs = block_sum<NTHR>(dot, red);
    double total;
    const unsigned nb = (unsigned)g.nit * g.njt * g.nkc;
    const unsigned blin = (unsigned)bx + g.nit * ((unsigned)by + g.njt * (unsigned)bz);
    if (last_block_sum_at<NTHR>(bs, a.partials, &a.st->cnt_a, nb, blin, &total, red)) {
      if (threadIdx.x == 0) {
        SolveState *s = a.st;
        s->pq = total;
        s->par = par ^ 1;
        if (!(total != 0.0) || !isfinite(total)) {
          s->status = ST_BREAKDOWN;
          s->alpha = 0.0;
        } else {
          s->alpha = s->rho / total;
        }
        if (a.xslot1) s->xa[a.xslot1 - 1] = s->alpha;
      }
    }
  }
}

// The PCGZ stages (one FP64 and one FP32 box per plane) and the PCGZ32
// stages (two FP32 boxes) fit three blocks per SM in shared memory, so those
// modes are compiled for three; the others hold more per stage and stay at
// two (a tighter register cap only slows them).
template <int MODE>
__global__ void __launch_bounds__(NTHR, (MODE == MODE_PCGZ || MODE == MODE_PCGZ32) ? 3 : 2)
    k_stencil(const __grid_constant__ StencilMaps maps, Geo g, DevMesh m, StencilArgs a) {
  stencil_body<MODE>(maps, g, m, a, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ============================================================================
// Update kernel: x += alpha p ; r -= alpha q ; z = a_i r ; rho = r.z
// (src/pot3d.F90:4344-4352) and ernorm (src/pot3d.F90:4430-4483) in the
// last block.  INIT: alpha = 0 and x, p, q untouched (the initial residual
// of cgsolve, src/pot3d.F90:4317-4330).  DOT_ONLY: rho = r.z with no
// update, for bdotb (src/pot3d.F90:4293-4298).
// ============================================================================
struct UpdateArgs {
  double *x;
  const double *p;
  double *r;
  const double *q;
  const float *ai;
  const float *z32;       // ILU(0) output (ifprec=2); ai is then unused
  float *r32;             // ifprec=2: FP32 copy of r for the sweeps; R32: the residual itself
  const float *p32;       // R32: FP32 search direction and A p
  const float *q32;
  double *s1z_part;       // [nkc][NRP]
  SolveState *st;
  double *partials;
};
// UPD_ZDOT: r.z with z from the ILU(0) sweeps, ncg+1 and ernorm, no update.
// UPD_RU: r.z of a freshly computed FP64 residual (a reliable update of the
// FP32-inner solve): rho and beta are replaced, ncg does not advance, and
// the status is decided on this residual whatever the recurrence said
// (rz_epilogue).

// R32: the residual (and, for UPD_ITER, p and q) are FP32 vectors; the
// arithmetic is FP64 and the new residual is rounded once when stored.
// X: UPD_ITER also updates x; without, x is left to k_update_x_group.
// S: planes whose loads are issued ahead of the first plane's stores.
template <int KIND, bool ZIN, bool R32, bool X, int S>
__device__ __forceinline__ void update_body(const Geo &g, const DevMesh &m, const UpdateArgs &a, const int bx,
                                            const int by, const int bz) {
  __shared__ double red[NTHR / 32];
  pdl_wait();
  pdl_trigger();
  const volatile SolveState *vs = a.st;
  if ((KIND == UPD_ITER || KIND == UPD_ZDOT) && vs->status != ST_RUNNING) return;
  const double alpha = (KIND == UPD_ITER) ? vs->alpha : 0.0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e0 = bx * TI + 2 * lane;
  const int jj = by * TJ + w;
  const int k0 = bz * g.tk_u;
  const int k1 = min(k0 + g.tk_u, g.npm2);
  const bool v0 = jj < g.ntm2 && e0 < g.nrm2;
  const bool v1 = v0 && e0 + 1 < g.nrm2;
  const bool south = v0 && jj == g.ntm2 - 1;
  double rz = 0.0, s1a = 0.0, s1b = 0.0;
  // r, q, p and z come from the kernels before: ordinary loads (see pdl_wait)
  using V = typename std::conditional<R32, float2, double2>::type;
  auto wide = [](V v) {
    if constexpr (R32)
      return widen2(v);
    else
      return v;
  };
  V *rv;
  const V *qv, *pv;
  if constexpr (R32) {
    rv = reinterpret_cast<V *>(a.r32);
    qv = reinterpret_cast<const V *>(a.q32);
    pv = reinterpret_cast<const V *>(a.p32);
  } else {
    rv = reinterpret_cast<V *>(a.r);
    qv = reinterpret_cast<const V *>(a.q);
    pv = reinterpret_cast<const V *>(a.p);
  }
  double2 *const xv = reinterpret_cast<double2 *>(a.x);
  const long long step = (long long)g.NRP * g.ntm2 / 2;
  auto planes = [&](auto nc, int kk) {
    constexpr int N = decltype(nc)::value;
    const long long id0 = g.idx(e0, jj, kk) / 2;
    V r0[N], q0[N], p0[N];
    double2 x0[N];
    float2 z0[N];
#pragma unroll
    for (int s = 0; s < N; s++) {
      const long long id = id0 + s * step;
      r0[s] = rv[id];
      if (KIND == UPD_ITER) q0[s] = qv[id];
      if (X) {
        x0[s] = xv[id];
        p0[s] = pv[id];
      }
      z0[s] = ZIN ? reinterpret_cast<const float2 *>(a.z32)[id] : __ldg(reinterpret_cast<const float2 *>(a.ai) + id);
    }
#pragma unroll
    for (int s = 0; s < N; s++) {
      const long long id = id0 + s * step;
      if (X) {
        const double2 p = wide(p0[s]);
        xv[id] = make_double2(fma(alpha, p.x, x0[s].x), fma(alpha, p.y, x0[s].y));
      }
      double2 r = wide(r0[s]);
      if (KIND == UPD_ITER) {
        const double2 q = wide(q0[s]);
        r.x = fma(-alpha, q.x, r.x);
        r.y = fma(-alpha, q.y, r.y);
        if constexpr (R32) {
          const float2 r2 = make_float2((float)r.x, (float)r.y);
          rv[id] = r2;
          r = widen2(r2);  // r.z of the stored residual
        } else {
          rv[id] = r;
        }
      }
      if (!v1) r.y = 0.0;
      const double zx = ZIN ? (double)z0[s].x : (double)z0[s].x * r.x;
      double zy = ZIN ? (double)z0[s].y : (double)z0[s].y * r.y;
      if (!v1) zy = 0.0;
      rz = fma(r.x, zx, rz);
      rz = fma(r.y, zy, rz);
      if (south && KIND != UPD_BDOTB) {
        const double wk = m.dph[kk + s + 2];
        s1a += __dmul_rn(zx, wk) * m.pl_i;
        s1b += __dmul_rn(zy, wk) * m.pl_i;
      }
    }
  };
  if (v0) {
    int kk = k0;
    if (S > 1)
      for (; kk + S <= k1; kk += S) planes(std::integral_constant<int, S>{}, kk);
#pragma unroll (S > 1 ? 1 : 4)
    for (; kk < k1; kk++) planes(std::integral_constant<int, 1>{}, kk);
  }
  if (south && KIND != UPD_BDOTB) {
    a.s1z_part[(long long)bz * g.NRP + e0] = s1a;
    if (e0 + 1 < g.NRP) a.s1z_part[(long long)bz * g.NRP + e0 + 1] = v1 ? s1b : 0.0;
  }
  const double bs = block_sum<NTHR>(rz, red);
  double total;
  const unsigned nb = (unsigned)g.nit * g.njt * g.nkc_u;
  const unsigned blin = (unsigned)bx + g.nit * ((unsigned)by + g.njt * (unsigned)bz);
  if (last_block_sum_at<NTHR>(bs, a.partials, &a.st->cnt_b, nb, blin, &total, red)) {
    if (threadIdx.x == 0) {
      SolveState *s = a.st;
      if (KIND == UPD_BDOTB) {
        s->bdotb = total;
      } else {
        rz_epilogue<KIND == UPD_BDOTB ? UPD_ITER : KIND>(s, total);
      }
    }
  }
}

// Planes ahead (S) and blocks an SM.  Ordinary loads do not pass the stores of
// the planes before, so a form says how many planes it loads first; with one
// plane at a time and 40 registers, as with the read-only loads it had, a solve
// took 6.04 s at 255x361x721 FP64, 455 ms at 121x181x361, 298 at 127x181x361
// refined, 33.3 at 63x91x181.  Without x: FP64 four planes and three blocks
// (5.87 s, 441 ms; 8 planes 5.99 and 449, 2 planes at six blocks 5.91 and 448),
// refined two and six (286 ms; 4 at four 295, 4 at five 309).  With x, on grids
// within L2: one plane, five blocks (32.0 ms; 2 planes 33.1).  Batches: two
// planes, four blocks (six grids of 63 to 127 x 91 to 181 x 181 to 361: 1194 ms
// FP64, 1042 refined; one plane 1193 and 1088).
constexpr int upd_planes(int kind, bool r32, bool x) { return kind != UPD_ITER || x ? 1 : r32 ? 2 : 4; }
constexpr int upd_blocks(int kind, bool r32, bool x) { return kind != UPD_ITER ? 6 : x ? 5 : r32 ? 6 : 3; }
template <int KIND, bool ZIN, bool R32 = false, bool X = KIND == UPD_ITER>
__global__ void __launch_bounds__(NTHR, upd_blocks(KIND, R32, X)) k_update(Geo g, DevMesh m, UpdateArgs a) {
  update_body<KIND, ZIN, R32, X, upd_planes(KIND, R32, X)>(g, m, a, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ifprec=2 half of the update: x += alpha p ; r -= alpha q ; r32 = (float)r
// (the FP64->FP32 cast of prec_inv, src/pot3d.F90:5207-5209, fused).
__device__ __forceinline__ void update_r32_body(const Geo &g, const UpdateArgs &a, long long t0, long long stride) {
  const volatile SolveState *vs = a.st;
  if (vs->status != ST_RUNNING) return;
  const double alpha = vs->alpha;
  const long long n = g.Np;
  for (long long t = t0; 2 * t < n; t += stride) {
    const long long id = 2 * t;
    double2 xv = *reinterpret_cast<const double2 *>(a.x + id);
    double2 rv = *reinterpret_cast<const double2 *>(a.r + id);
    const double2 pv = __ldg(reinterpret_cast<const double2 *>(a.p + id));
    const double2 qv = __ldg(reinterpret_cast<const double2 *>(a.q + id));
    xv.x = fma(alpha, pv.x, xv.x);
    xv.y = fma(alpha, pv.y, xv.y);
    rv.x = fma(-alpha, qv.x, rv.x);
    rv.y = fma(-alpha, qv.y, rv.y);
    *reinterpret_cast<double2 *>(a.x + id) = xv;
    *reinterpret_cast<double2 *>(a.r + id) = rv;
    *reinterpret_cast<float2 *>(a.r32 + id) = make_float2((float)rv.x, (float)rv.y);
  }
}
__global__ void __launch_bounds__(NTHR) k_update_r32(Geo g, UpdateArgs a) {
  update_r32_body(g, a, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}
__global__ void k_cast_r32(long long n, const double *__restrict__ r, float *__restrict__ r32) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    r32[t] = (float)r[t];
}

// ============================================================================
// FP32-inner / FP64-refined PCG (both preconditioners).  The inner
// iterations keep p, q and the recurrence residual r in FP32 (half the bytes
// of the FP64 iteration) while every product is formed in FP64 registers:
// the stencil (MODE_PCG32 / MODE_PCGZ32), alpha, beta and the dots
// (accumulated in FP64), and the solution update x += alpha p on the FP64 x.
// A reliable update recomputes r = b - A x in FP64 and its preconditioned
// norm (the reference's epsn, src/pot3d.F90:4432-4433), replaces the
// recurrence's rho with it and keeps the search direction; convergence is
// only ever accepted on that FP64 residual.
// ============================================================================

// Solution half of the refined ILU(0) inner update (the residual half,
// r32 = r32 - alpha q rounded once, runs inside the forward sweep, which
// reads the residual), applied to groups of iterations: x += alpha_a p_a,
// then x += alpha_b p_b, with p_a, p_b the search directions of two
// consecutive iterations, which the ping-pong buffers still hold, and the
// alphas their stencils recorded in st->xa (0 for an iteration that did not
// run).  One fma of FP64 x with the FP32 direction per point and iteration,
// in iteration order, so x is bit-identical to updating it every iteration,
// and the solution vector is read and written once per group.  Four
// unknowns per thread and pass.  Batches use pairs; single solves larger groups
// (k_update_x_group).
__device__ __forceinline__ void x_pair_body(const Geo &g, const SolveState *st, double *__restrict__ x,
                                            const float *__restrict__ pa, const float *__restrict__ pb, long long t0,
                                            long long stride) {
  const double a0 = *(const volatile double *)&st->xa[0], a1 = *(const volatile double *)&st->xa[1];
  if (a0 == 0.0 && a1 == 0.0) return;
  const long long n4 = g.Np / 4;
  for (long long t = t0; t < n4; t += stride) {
    const long long id = 4 * t;
    double2 x0 = *reinterpret_cast<const double2 *>(x + id);
    double2 x1 = *reinterpret_cast<const double2 *>(x + id + 2);
    const float4 u = __ldg(reinterpret_cast<const float4 *>(pa + id));
    const float4 v = __ldg(reinterpret_cast<const float4 *>(pb + id));
    if (a0 != 0.0) {
      x0.x = fma(a0, (double)u.x, x0.x);
      x0.y = fma(a0, (double)u.y, x0.y);
      x1.x = fma(a0, (double)u.z, x1.x);
      x1.y = fma(a0, (double)u.w, x1.y);
    }
    if (a1 != 0.0) {
      x0.x = fma(a1, (double)v.x, x0.x);
      x0.y = fma(a1, (double)v.y, x0.y);
      x1.x = fma(a1, (double)v.z, x1.x);
      x1.y = fma(a1, (double)v.w, x1.y);
    }
    *reinterpret_cast<double2 *>(x + id) = x0;
    *reinterpret_cast<double2 *>(x + id + 2) = x1;
  }
}
// The single solves' groups: G iterations at once, x += a_0 p_0 + ... +
// a_{G-1} p_{G-1} in iteration order (the directions of G consecutive
// iterations, in the rotating buffers), x read and written once per group.
// With FP32 directions and G = 8 this moves 6 B per unknown and iteration
// instead of 20, with FP64 directions and G = 4 12 B instead of 24: the
// 121x181x361 FP64 solve spent 73 us of 134 us an iteration in an update that
// read and wrote x every time.
template <typename T, int G>
struct XDirs {
  const T *p[G];
};
template <typename T, int G>
__global__ void __launch_bounds__(NTHR) k_update_x_group(Geo g, const SolveState *st, double *__restrict__ x,
                                                         XDirs<T, G> d) {
  pdl_wait();
  pdl_trigger();
  double a[G];
  bool any = false;
#pragma unroll
  for (int i = 0; i < G; i++) {
    a[i] = *(const volatile double *)&st->xa[i];
    any = any || a[i] != 0.0;
  }
  if (!any) return;
  const long long n4 = g.Np / 4;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n4;
       t += (long long)gridDim.x * blockDim.x) {
    const long long id = 4 * t;
    double2 x0 = *reinterpret_cast<const double2 *>(x + id);
    double2 x1 = *reinterpret_cast<const double2 *>(x + id + 2);
    double2 v0[G], v1[G];
#pragma unroll
    for (int i = 0; i < G; i++) {
      if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(d.p[i] + id);
        v0[i] = make_double2((double)v.x, (double)v.y);
        v1[i] = make_double2((double)v.z, (double)v.w);
      } else {
        v0[i] = *reinterpret_cast<const double2 *>(d.p[i] + id);
        v1[i] = *reinterpret_cast<const double2 *>(d.p[i] + id + 2);
      }
    }
#pragma unroll
    for (int i = 0; i < G; i++) {
      if (a[i] != 0.0) {
        x0.x = fma(a[i], v0[i].x, x0.x);
        x0.y = fma(a[i], v0[i].y, x0.y);
        x1.x = fma(a[i], v1[i].x, x1.x);
        x1.y = fma(a[i], v1[i].y, x1.y);
      }
    }
    *reinterpret_cast<double2 *>(x + id) = x0;
    *reinterpret_cast<double2 *>(x + id + 2) = x1;
  }
}

// South-ring partial sums of z for the next stencil after the fused sweeps
// (which leave no r.z kernel to form them): s1z_part[c][e] = sum over the
// planes of k chunk c of z(e, ntm1, k)*dph(k)*pl_i, in update_body's order.
__device__ __forceinline__ void south_ring_z_body(const Geo &g, const DevMesh &m, const float *__restrict__ z32,
                                                  double *__restrict__ s1z_part, int e, int bz) {
  if (e >= g.nrm2) return;
  const int k0 = bz * g.tk_u, k1 = min(k0 + g.tk_u, g.npm2);
  double s1 = 0.0;
#pragma unroll 8  // the loads of a block of planes issue together; the sum keeps its order
  for (int kk = k0; kk < k1; kk++) {
    const double zx = z32[g.idx(e, g.ntm2 - 1, kk)];
    s1 += __dmul_rn(zx, m.dph[kk + 2]) * m.pl_i;
  }
  s1z_part[(long long)bz * g.NRP + e] = s1;
}
__global__ void k_south_ring_z(Geo g, DevMesh m, const float *__restrict__ z32, double *__restrict__ s1z_part) {
  south_ring_z_body(g, m, z32, s1z_part, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y);
}

// r = b - q (the FP64 true residual of a reliable update, q = A x) and its
// FP32 copy for the inner iterations and the sweeps.
__global__ void k_resid_cast(long long n, const double *__restrict__ b, const double *__restrict__ q,
                             double *__restrict__ r, float *__restrict__ r32) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double v = b[t] - q[t];
    r[t] = v;
    r32[t] = (float)v;
  }
}

// ============================================================================
// Small kernels: layout conversion, ring sums, RHS, phi finalisation,
// energies, plain dots.
// ============================================================================
__global__ void k_pack(Geo g, const double *__restrict__ src, double *__restrict__ dst) {
  // reference packed layout -> padded layout (zeros in the pad lanes)
  const long long n = g.Np;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t % g.NRP);
    const long long line = t / g.NRP;
    dst[t] = (e < g.nrm2) ? src[line * g.nrm2 + e] : 0.0;
  }
}
__global__ void k_unpack(Geo g, const double *__restrict__ src, double *__restrict__ dst) {
  const long long n = g.N;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t % g.nrm2);
    const long long line = t / g.nrm2;
    dst[t] = src[line * g.NRP + e];
  }
}
// S1(e) = sum_k x(e, ntm1, k)*dph(k)*pl_i in k order (src/pot3d.F90:5456-5463).
// A block takes 32 radial points, its 32 warps 32 planes at a time, so the
// loads are in flight together; the sum keeps the planes' order.  (One thread
// walking a radial point's planes alone took 130 us at 127x181x361.)
__global__ void __launch_bounds__(1024) k_ring_south(Geo g, DevMesh m, const double *__restrict__ x,
                                                     double *__restrict__ s1) {
  __shared__ double t[32][33];
  const int lane = threadIdx.x & 31, y = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double s = 0.0;
  for (int k0 = 0; k0 < g.npm2; k0 += 32) {
    const int kk = k0 + y;
    t[y][lane] = e < g.nrm2 && kk < g.npm2
                     ? __dmul_rn(__dmul_rn(x[g.idx(e, g.ntm2 - 1, kk)], m.dph[kk + 2]), m.pl_i)
                     : 0.0;
    __syncthreads();
    if (y == 0) {
      const int n = min(32, g.npm2 - k0);
      for (int q = 0; q < n; q++) s = s + t[q][lane];
    }
    __syncthreads();
  }
  if (y == 0 && e < g.NRP) s1[e] = s;
}
// RHS of the boundary trick, src/pot3d.F90:3937-3950: with a zero interior,
// delsq at i=2 picks up a3*x(1) where x(1) = -br0*dr1 and, for a
// validation run, a5*x(nr) at i=nrm1 where x(nr) = br1*drn; every other
// term multiplies an exact zero.  rhs = -delsq.
__global__ void k_rhs(Geo g, DevMesh m, double *__restrict__ rhs) {
  const long long n = g.Np;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t % g.NRP);
    const long long line = t / g.NRP;
    const int jj = (int)(line % g.ntm2), kk = (int)(line / g.ntm2);
    double v = 0.0;
    if (e < g.nrm2 && (e == 0 || (m.br1 && e == g.nrm2 - 1))) {
      const int i = e + 2, j = jj + 2, k = kk + 2;
      const RowCoef rc = row_coef(m, j);
      const PtCoef pc = pt_coef(m, i, j);
      const Coef7 c = coef7(pc, rc, m.dp_i[k - 1], m.dp_i[k], m.dph[k]);
      double y = 0.0;
      if (e == 0) {
        const double x1 = -__dmul_rn(m.br0[(j - 1) + (long long)g.nt * (k - 1)], m.dr1);
        y = c.a3 * x1;
      }
      if (m.br1 && e == g.nrm2 - 1) {
        const double xn = __dmul_rn(m.br1[(j - 1) + (long long)g.nt * (k - 1)], m.drn);
        y = fma(c.a5, xn, y);
      }
      v = -y;
    }
    rhs[t] = v;
  }
}
// Unpack x into phi(nr,nt,np) and set the radial ghosts with vmask=1.
__global__ void k_phi_interior(Geo g, DevMesh m, const double *__restrict__ xpad, double *__restrict__ phi) {
  const long long n = (long long)g.nr * g.nt * g.np;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % g.nr) + 1;
    const int j = (int)((t / g.nr) % g.nt) + 1;
    const int k = (int)(t / ((long long)g.nr * g.nt)) + 1;
    double v = 0.0;
    const bool jin = j >= 2 && j <= g.nt - 1, kin = k >= 2 && k <= g.np - 1;
    if (jin && kin) {
      const int ic = (i == 1) ? 2 : (i == g.nr ? g.nr - 1 : i);
      const double xi = xpad[g.idx(ic - 2, j - 2, k - 2)];
      if (i == 1) {
        v = xi - __dmul_rn(m.br0[(j - 1) + (long long)g.nt * (k - 1)], m.dr1);
      } else if (i == g.nr) {
        v = m.br1 ? xi + __dmul_rn(m.br1[(j - 1) + (long long)g.nt * (k - 1)], m.drn) : m.pm_r1 * xi;
      } else {
        v = xi;
      }
    }
    phi[t] = v;
  }
}
// Pole ring sums over phi, i = 1..nr, in k order (src/pot3d.F90:5442-5465).
__global__ void k_phi_ring(Geo g, DevMesh m, const double *__restrict__ phi, double *__restrict__ sums) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > g.nr) return;
  const long long pl = (long long)g.nr * g.nt;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll 16
  for (int k = 2; k <= g.np - 1; k++) {
    s0 = s0 + __dmul_rn(__dmul_rn(phi[(i - 1) + (long long)g.nr * 1 + pl * (k - 1)], m.dph[k]), m.pl_i);
    s1 = s1 + __dmul_rn(__dmul_rn(phi[(i - 1) + (long long)g.nr * (g.nt - 2) + pl * (k - 1)], m.dph[k]), m.pl_i);
  }
  sums[2 * i] = s0;
  sums[2 * i + 1] = s1;
}
__global__ void k_phi_poles(Geo g, const double *__restrict__ sums, double *__restrict__ phi) {
  const long long n = (long long)g.nr * (g.np - 2);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % g.nr) + 1;
    const int k = (int)(t / g.nr) + 2;
    const long long pl = (long long)g.nr * g.nt;
    const long long b = (i - 1) + pl * (k - 1);
    phi[b] = 2.0 * sums[2 * i] - phi[b + g.nr];
    phi[b + (long long)g.nr * (g.nt - 1)] = 2.0 * sums[2 * i + 1] - phi[b + (long long)g.nr * (g.nt - 2)];
  }
}
__global__ void k_phi_seam(Geo g, double *__restrict__ phi) {
  const long long pl = (long long)g.nr * g.nt;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < pl;
       t += (long long)gridDim.x * blockDim.x) {
    phi[t] = phi[t + pl * (g.np - 2)];
    phi[t + pl * (g.np - 1)] = phi[t + pl];
  }
}
// getb + magnetic_energy fused (src/pot3d.F90:6217-6231, 6279-6292).
__global__ void __launch_bounds__(NTHR) k_energy(Geo g, DevMesh m, const double *__restrict__ phi,
                                                 double *__restrict__ part) {
  __shared__ double red[NTHR / 32];
  const long long nint = (long long)(g.nr - 2) * (g.nt - 2) * (g.np - 2);
  double wr = 0.0, wt = 0.0, wp = 0.0;
  const long long nr = g.nr, ntr = (long long)g.nr * g.nt;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nint;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t % (g.nr - 2)) + 2;
    const int j = (int)((t / (g.nr - 2)) % (g.nt - 2)) + 2;
    const int k = (int)(t / ((long long)(g.nr - 2) * (g.nt - 2))) + 2;
    const long long c = (i - 1) + nr * (j - 1) + ntr * (k - 1);
    const double f = phi[c];
    const double br_p = (phi[c + 1] - f) / m.dr[i];
    const double br_m = (f - phi[c - 1]) / m.dr[i - 1];
    const double rhi = m.rh[i];
    const double bt_p = (phi[c + nr] - f) / (rhi * m.dt[j]);
    const double bt_m = (f - phi[c - nr]) / (rhi * m.dt[j - 1]);
    const double bp_p = (phi[c + ntr] - f) / (__dmul_rn(rhi, m.sth[j]) * m.dp[k]);
    const double bp_m = (f - phi[c - ntr]) / (__dmul_rn(rhi, m.sth[j]) * m.dp[k - 1]);
    const double dv = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(rhi, rhi), m.drh[i]), m.dth[j]), m.sth[j]),
                                m.dph[k]);
    const double brav = 0.5 * (br_p + br_m);
    const double btav = 0.5 * (bt_p + bt_m);
    const double bpav = 0.5 * (bp_p + bp_m);
    wr += __dmul_rn(0.5 * __dmul_rn(brav, brav), dv);
    wt += __dmul_rn(0.5 * __dmul_rn(btav, btav), dv);
    wp += __dmul_rn(0.5 * __dmul_rn(bpav, bpav), dv);
  }
  double s0 = block_sum<NTHR>(wr, red);
  double s1 = block_sum<NTHR>(wt, red);
  double s2 = block_sum<NTHR>(wp, red);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x + 0] = s0;
    part[3 * blockIdx.x + 1] = s1;
    part[3 * blockIdx.x + 2] = s2;
  }
}
// getb, src/pot3d.F90:6187-6233: one pass over phi writes every point the
// reference fills of the three staggered components, br (nrm1,nt,np),
// bt (nr,ntm1,np) and bp (nr,nt,npm1), column-major.  The denominators'
// products round left to right, as in the Fortran.
__global__ void __launch_bounds__(NTHR) k_getb(Geo g, DevMesh m, const double *__restrict__ phi,
                                               double *__restrict__ br, double *__restrict__ bt,
                                               double *__restrict__ bp) {
  const long long nr = g.nr, nt = g.nt, ntr = nr * nt, n = ntr * g.np;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
       c += (long long)gridDim.x * blockDim.x) {
    const int i0 = (int)(c % nr);
    const long long jk = c / nr;
    const int j0 = (int)(jk % nt);
    const int k0 = (int)(jk / nt);
    const double f = phi[c];
    const double rhi = m.rh[i0 + 1];
    if (i0 < g.nr - 1) br[i0 + (nr - 1) * jk] = (phi[c + 1] - f) / m.dr[i0 + 1];
    if (j0 < g.nt - 1)
      bt[i0 + nr * (j0 + (nt - 1) * (long long)k0)] = (phi[c + nr] - f) / __dmul_rn(rhi, m.dt[j0 + 1]);
    if (k0 < g.np - 1) bp[c] = (phi[c + ntr] - f) / __dmul_rn(__dmul_rn(rhi, m.sth[j0 + 1]), m.dp[k0 + 1]);
  }
}
__global__ void k_energy_final(const double *__restrict__ part, int nb, double *__restrict__ w) {
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp a component; a fixed order
  double s = 0.0;
#pragma unroll 8
  for (int b = lane; b < nb; b += 32) s += part[3 * b + c];
  s = warp_sum(s);
  if (lane == 0) w[c] = s;
}
// Deterministic dot of two padded vectors (two-stage).
__global__ void __launch_bounds__(NTHR) k_dot(long long n, const double *__restrict__ x,
                                              const double *__restrict__ y, double *__restrict__ part) {
  __shared__ double red[NTHR / 32];
  double s = 0.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    s = fma(x[t], y[t], s);
  s = block_sum<NTHR>(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}
__global__ void k_sum_parts(const double *__restrict__ part, int nb, double *__restrict__ out) {
  double s = 0.0;  // one warp; a fixed order
#pragma unroll 8
  for (int b = threadIdx.x; b < nb; b += 32) s += part[b];
  s = warp_sum(s);
  if (threadIdx.x == 0) *out = s;
}
__global__ void k_axpy_sub(long long n, const double *__restrict__ q, double *__restrict__ r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    r[t] = r[t] - q[t];
}
// a_i = real(1/a(i,j,k,4), REAL32), src/pot3d.F90:4653-4661.
__global__ void k_diag_prec(Geo g, DevMesh m, float *__restrict__ ai, int ifprec) {
  const long long n = g.Np;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t % g.NRP);
    const long long line = t / g.NRP;
    const int jj = (int)(line % g.ntm2), kk = (int)(line / g.ntm2);
    float v = 0.0f;
    if (e < g.nrm2) {
      if (ifprec == 0) {
        v = 1.0f;
      } else {
        const int i = e + 2, j = jj + 2, k = kk + 2;
        const Coef7 c = coef7(pt_coef(m, i, j), row_coef(m, j), m.dp_i[k - 1], m.dp_i[k], m.dph[k]);
        v = __double2float_rn(__ddiv_rn(1.0, c.a4));
      }
    }
    ai[t] = v;
  }
}
__global__ void k_widen(long long n, const float *__restrict__ z, double *__restrict__ x) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    x[t] = (double)z[t];
}
__global__ void k_scale_ai(long long n, const float *__restrict__ ai, double *__restrict__ x) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    x[t] = (double)ai[t] * x[t];
}


// ============================================================================
// Host side of the FP64 solver.
// ============================================================================
namespace pot3d {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 3-D tensor map of a padded vector (i, j, k) = (NRP, ntm2, npm2) with a
// box of bx x by x bz elements; zero fill outside the vector.
int encode_padded_map(const Geo &g, const void *ptr, bool fp64, int bx, int by, int bz, CUtensorMap *out,
                      bool interior_only) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) {
    pot3d_set_error("cuTensorMapEncodeTiled is not available from the driver");
    return POT3D_ERR_CUDA;
  }
  const cuuint64_t es = fp64 ? 8 : 4;
  // interior_only: the map ends at e = nrm2, so a store through it never
  // writes the padding columns of a line
  cuuint64_t dims[3] = {(cuuint64_t)(interior_only ? g.nrm2 : g.NRP), (cuuint64_t)g.ntm2, (cuuint64_t)g.npm2};
  cuuint64_t strides[2] = {(cuuint64_t)g.NRP * es, (cuuint64_t)g.NRP * g.ntm2 * es};
  cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bz};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, fp64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                  const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    pot3d_set_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
    return POT3D_ERR_CUDA;
  }
  return POT3D_OK;
}

// 3-D tensor map of a padded vector (i, j, k) = (NRP, ntm2, npm2) with the
// stencil's box: 68 x 10 x 1 FP64 or 72 x 10 x 1 FP32.
int Solver::tensor_map(const void *ptr, bool fp64, CUtensorMap *out) {
  auto key = std::make_pair(ptr, fp64 ? 1 : 0);
  auto it = tmaps.find(key);
  if (it != tmaps.end()) {
    *out = it->second;
    return POT3D_OK;
  }
  EncodeTiledFn fn = encode_tiled();
  if (!fn) {
    pot3d_set_error("cuTensorMapEncodeTiled is not available from the driver");
    return POT3D_ERR_CUDA;
  }
  const cuuint64_t es = fp64 ? 8 : 4;
  cuuint64_t dims[3] = {(cuuint64_t)g.NRP, (cuuint64_t)g.ntm2, (cuuint64_t)g.npm2};
  cuuint64_t strides[2] = {(cuuint64_t)g.NRP * es, (cuuint64_t)g.NRP * g.ntm2 * es};
  cuuint32_t box[3] = {(cuuint32_t)(fp64 ? BOX64_X : BOX32_X), (cuuint32_t)BOX_Y, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap mp;
  CUresult r = fn(&mp, fp64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                  const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    pot3d_set_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
    return POT3D_ERR_CUDA;
  }
  tmaps[key] = mp;
  *out = mp;
  return POT3D_OK;
}

template <int MODE>
static int set_stencil_smem() {
  return pot3d_cuda_status(cudaFuncSetAttribute(k_stencil<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                StageLayout<MODE>::smem),
                           "cudaFuncSetAttribute(k_stencil)");
}

int grid1d(long long n) {
  long long b = (n + NTHR - 1) / NTHR;
  if (b > 148LL * 16) b = 148LL * 16;
  if (b < 1) b = 1;
  return (int)b;
}

static double *upload_1based(const double *src, int n, Solver *s, int *st) {
  std::vector<double> h(n + 2, 0.0);
  for (int q = 0; q < n; q++) h[q + 1] = src[q];
  double *d = nullptr;
  int e = s->alloc((void **)&d, sizeof(double) * (n + 2));
  if (e) {
    *st = e;
    return nullptr;
  }
  e = pot3d_cuda_status(cudaMemcpy(d, h.data(), sizeof(double) * (n + 2), cudaMemcpyHostToDevice),
                        "cudaMemcpy(mesh)");
  if (e) *st = e;
  return d;
}

int Solver::alloc(void **p, size_t bytes) {
  *p = nullptr;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) return pot3d_cuda_status(e, "cudaMalloc");
  allocs.push_back(*p);
  e = cudaMemset(*p, 0, bytes);
  return pot3d_cuda_status(e, "cudaMemset");
}

Solver::~Solver() {
  if (stream) cudaStreamSynchronize(stream);
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  if (dilu) dilu_destroy(this);
  if (graph32_exec) cudaGraphExecDestroy(graph32_exec);
  if (evm0) cudaEventDestroy(evm0);
  if (evm1) cudaEventDestroy(evm1);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);

  for (void *p : allocs) cudaFree(p);
  if (h_state) cudaFreeHost(h_state);
  if (stream) cudaStreamDestroy(stream);
}

int Solver::setup(const pot3d_mesh_t *mesh, const double *br0, const double *br1, double pm_r1_,
                  int ifprec_, int precision_) {
  const int nr = mesh->nr, nt = mesh->nt, np = mesh->np;
  if (nr < 4 || nt < 5 || np < 6) {
    pot3d_set_error("mesh too small: need nr>=4, nt>=5, np>=6");
    return POT3D_ERR_ARG;
  }
  if (ifprec_ < 0 || ifprec_ > 2 || precision_ < 0 || precision_ > 1) {
    pot3d_set_error("invalid ifprec or precision mode");
    return POT3D_ERR_ARG;
  }
  if (mesh->st[0] != 0.0) {
    pot3d_set_error("st(1) must be sin(0)=0: the theta mesh starts at the pole");
    return POT3D_ERR_ARG;
  }
  ifprec = ifprec_;
  precision = precision_;
  // With br1 (a validation run) the r=R1 ghost is x(nr) = x(nrm1) +
  // vmask*br1*drn (src/pot3d.F90:5420-5423): the operator's homogeneous part
  // (vmask = 0) couples x(nr) to x(nrm1) with factor +1 whatever the option.
  pm_r1 = br1 ? 1.0 : pm_r1_;
  g.nr = nr;
  g.nt = nt;
  g.np = np;
  g.nrm2 = nr - 2;
  g.ntm2 = nt - 2;
  g.npm2 = np - 2;
  g.NRP = (g.nrm2 + 15) / 16 * 16;
  g.N = (long long)g.nrm2 * g.ntm2 * g.npm2;
  g.Np = (long long)g.NRP * g.ntm2 * g.npm2;
  g.nit = (g.nrm2 + TI - 1) / TI;
  g.njt = (g.ntm2 + TJ - 1) / TJ;

  // A blocking stream: ordered with the legacy default stream, where callers
  // (the Fortran host, torch) produce their device arrays and cudaMemset runs.
  CK(cudaStreamCreate(&stream));
  {
    int e;
    if ((e = set_stencil_smem<MODE_AX>()) || (e = set_stencil_smem<MODE_PCG>()) ||
        (e = set_stencil_smem<MODE_PCGZ>()) || (e = set_stencil_smem<MODE_PCG32>()) ||
        (e = set_stencil_smem<MODE_PCGZ32>()))
      return e;
  }
  // k-chunking by a wave model: the grid is (i tiles, j tiles, k chunks);
  // pick the chunk count that minimises whole waves x planes per block,
  // counting each block's pipeline start-up as extra planes.
  {
    int dev = 0, nsm = 148, occ_s = 2;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    // occupancy of the stencil form this solver iterates with (the ILU(0)
    // forms hold three blocks per SM, the diagonal ones two)
    if (ifprec == 2 && precision == POT3D_FP32_REFINED)
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, k_stencil<MODE_PCGZ32>, NTHR,
                                                       StageLayout<MODE_PCGZ32>::smem));
    else if (ifprec == 2)
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, k_stencil<MODE_PCGZ>, NTHR, StageLayout<MODE_PCGZ>::smem));
    else if (precision == POT3D_FP32_REFINED)
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, k_stencil<MODE_PCG32>, NTHR,
                                                       StageLayout<MODE_PCG32>::smem));
    else
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, k_stencil<MODE_PCG>, NTHR, StageLayout<MODE_PCG>::smem));
    const long long cols = (long long)g.nit * g.njt;
    auto pick = [&](int slots_per_sm, double startup, int max_tk, int *tk, int *nkc) {
      const double slots = (double)std::max(1, slots_per_sm) * nsm;
      double best = 1e300;
      for (int c = 1; c <= g.npm2; c++) {
        const int t = (g.npm2 + c - 1) / c;
        if (t > max_tk) continue;
        const int cc = (g.npm2 + t - 1) / t;
        const double waves = std::ceil((double)(cols * cc) / slots);
        const double cost = waves * (t + startup);
        if (cost < best - 1e-9) {
          best = cost;
          *tk = t;
          *nkc = cc;
        }
      }
    };
    pick(occ_s, 6.0, MAX_TK, &g.tk, &g.nkc);
    pick(6, 2.0, 1 << 30, &g.tk_u, &g.nkc_u);  // six blocks for every form: the order of r.z is the same in all
  }
  CK(cudaEventCreate(&ev0));
  CK(cudaEventCreate(&ev1));
  {
    int dev = 0, nsm = 148;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    xblocks = (int)std::min<long long>((g.Np / 4 + NTHR - 1) / NTHR, 8LL * nsm);
  }
  int st = POT3D_OK;
  std::vector<double> r2(nr - 1), dr_i(nr - 1), sth_i(nt), dt_i(nt - 1), dp_i(np);
  for (int i = 0; i < nr - 1; i++) {  // set_local_mesh_r, src/pot3d.F90:2752-2756
    r2[i] = mesh->r[i] * mesh->r[i];
    dr_i[i] = 1.0 / mesh->dr[i];
  }
  for (int j = 0; j < nt; j++) sth_i[j] = 1.0 / mesh->sth[j];  // src/pot3d.F90:2836-2840
  for (int j = 0; j < nt - 1; j++) dt_i[j] = 1.0 / mesh->dt[j];
  for (int k = 0; k < np; k++) dp_i[k] = 1.0 / mesh->dp[k];
  m.drh = upload_1based(mesh->drh, nr, this, &st);
  m.dth = upload_1based(mesh->dth, nt, this, &st);
  m.sth_i = upload_1based(sth_i.data(), nt, this, &st);
  m.dp_i = upload_1based(dp_i.data(), np, this, &st);
  m.dph = upload_1based(mesh->dph, np, this, &st);
  m.st = upload_1based(mesh->st, nt - 1, this, &st);
  m.dt_i = upload_1based(dt_i.data(), nt - 1, this, &st);
  m.sth = upload_1based(mesh->sth, nt, this, &st);
  m.r2 = upload_1based(r2.data(), nr - 1, this, &st);
  m.dr_i = upload_1based(dr_i.data(), nr - 1, this, &st);
  m.dr = upload_1based(mesh->dr, nr - 1, this, &st);
  m.rh = upload_1based(mesh->rh, nr, this, &st);
  m.dt = upload_1based(mesh->dt, nt - 1, this, &st);
  m.dp = upload_1based(mesh->dp, np, this, &st);
  m.th = upload_1based(mesh->th, nt, this, &st);
  m.ph = upload_1based(mesh->ph, np, this, &st);
  if (st != POT3D_OK) return st;
  m.dr1 = mesh->dr[0];
  m.drn = mesh->dr[nr - 2];
  m.pm_r1 = pm_r1;
  m.pl_i = 1.0 / (2.0 * 3.1415926535897932 - 0.0);
  const size_t nf = (size_t)nt * np;
  double *d_br0 = nullptr, *d_br1 = nullptr;
  if ((st = alloc((void **)&d_br0, nf * sizeof(double)))) return st;
  CK(cudaMemcpy(d_br0, br0, nf * sizeof(double), cudaMemcpyHostToDevice));
  if (br1) {
    if ((st = alloc((void **)&d_br1, nf * sizeof(double)))) return st;
    CK(cudaMemcpy(d_br1, br1, nf * sizeof(double), cudaMemcpyHostToDevice));
  }
  m.br0 = d_br0;
  m.br1 = d_br1;

  if ((st = alloc((void **)&d_state, sizeof(SolveState)))) return st;
  CK(cudaMallocHost(&h_state, sizeof(SolveState)));
  nblk_tiled = (size_t)g.nit * g.njt * std::max(g.nkc, g.nkc_u);
  if ((st = alloc((void **)&d_partials, sizeof(double) * std::max<size_t>(nblk_tiled, 148 * 16 * 3)))) return st;
  if ((st = alloc((void **)&d_s1z, sizeof(double) * (size_t)g.nkc_u * g.NRP))) return st;
  if ((st = alloc((void **)&d_s1p, sizeof(double) * 2 * (size_t)g.NRP))) return st;
  if ((st = alloc((void **)&d_s1, sizeof(double) * (size_t)g.NRP))) return st;
  if ((st = alloc((void **)&d_scalar, sizeof(double) * 8))) return st;
  if ((st = alloc((void **)&d_sums, sizeof(double) * 2 * (nr + 2)))) return st;
  hist_cap = 1 << 20;
  if ((st = alloc((void **)&d_hist, sizeof(double) * hist_cap))) return st;

  const size_t vb = sizeof(double) * (size_t)g.Np;
  if ((st = alloc((void **)&d_x, vb))) return st;
  if ((st = alloc((void **)&d_r, vb))) return st;
  if ((st = alloc((void **)&d_p, vb))) return st;
  if ((st = alloc((void **)&d_p2, vb))) return st;
  if ((st = alloc((void **)&d_q, vb))) return st;
  if ((st = alloc((void **)&d_b, vb))) return st;
  if ((st = alloc((void **)&d_tmp, vb))) return st;
  if (!batched) {  // host vectors' staging
    const size_t n1 = ((size_t)g.N + 31) / 32 * 32;
    if ((st = alloc((void **)&d_io, sizeof(double) * (n1 + (size_t)g.N)))) return st;
    d_io2 = d_io + n1;
  }
  if ((st = alloc((void **)&d_ai, sizeof(float) * (size_t)g.Np))) return st;
  k_diag_prec<<<grid1d(g.Np), NTHR, 0, stream>>>(g, m, d_ai, ifprec == 0 ? 0 : 1);
  CK(cudaGetLastError());
  if ((st = rhs_padded(d_b))) return st;
  if (ifprec == 2) {
    if ((st = dilu_setup(this))) return st;
  }
  if (precision == POT3D_FP32_REFINED) {
    const size_t fb = sizeof(float) * (size_t)g.Np;
    if ((st = alloc((void **)&m_p32a, fb)) || (st = alloc((void **)&m_p32b, fb)) || (st = alloc((void **)&m_q32, fb)))
      return st;
    if (ifprec != 2 && (st = alloc((void **)&m_r32, fb))) return st;  // ILU(0) uses the sweeps' r32
    CK(cudaEventCreate(&evm0));
    CK(cudaEventCreate(&evm1));
  }
  if ((st = x_buffers())) return st;
  CK(cudaStreamSynchronize(stream));
  return POT3D_OK;
}

int Solver::rhs_padded(double *b) {
  k_rhs<<<grid1d(g.Np), NTHR, 0, stream>>>(g, m, b);
  return pot3d_cuda_status(cudaGetLastError(), "k_rhs");
}

// y = A x on padded device vectors with the exact south-pole ring sums.
int Solver::ax_padded(const double *x, double *y) {
  k_ring_south<<<(g.NRP + 31) / 32, 1024, 0, stream>>>(g, m, x, d_s1);
  StencilArgs a{};
  a.x = x;
  a.y = y;
  a.s1_direct = d_s1;
  StencilMaps mp;
  int st;
  if ((st = tensor_map(x, true, &mp.m64[0]))) return st;
  mp.m64[1] = mp.m64[0];
  mp.m32[0] = mp.m32[1] = mp.m32[2] = mp.m64[0];
  dim3 grid(g.nit, g.njt, g.nkc);
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  k_stencil<MODE_AX><<<grid, NTHR, StageLayout<MODE_AX>::smem, stream>>>(mp, g, m, a);
  return pot3d_cuda_status(cudaGetLastError(), "k_stencil<AX>");
}

int Solver::prec_padded(double *x) {
  if (ifprec == 2) {
    k_cast_r32<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, x, dilu_r32(this));
    int st = dilu_sweeps(this, false);
    if (st || (st = dilu_status(this))) return st;
    // x = (double)z32
    k_widen<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, dilu_z32(this), x);
  } else {
    k_scale_ai<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_ai, x);
  }
  return pot3d_cuda_status(cudaGetLastError(), "prec");
}

int Solver::dot_padded(const double *x, const double *y, double *out_dev) {
  const int nb = 148 * 4;
  k_dot<<<nb, NTHR, 0, stream>>>(g.Np, x, y, d_partials);
  k_sum_parts<<<1, 32, 0, stream>>>(d_partials, nb, out_dev);
  return pot3d_cuda_status(cudaGetLastError(), "k_dot");
}

int Solver::pack(const double *ref_dev, double *pad_dev) {
  k_pack<<<grid1d(g.Np), NTHR, 0, stream>>>(g, ref_dev, pad_dev);
  return pot3d_cuda_status(cudaGetLastError(), "k_pack");
}
int Solver::unpack(const double *pad_dev, double *ref_dev) {
  k_unpack<<<grid1d(g.N), NTHR, 0, stream>>>(g, pad_dev, ref_dev);
  return pot3d_cuda_status(cudaGetLastError(), "k_unpack");
}

// The rotation of direction buffers (xg, xg64).  With the diagonal
// preconditioner x is updated in groups where the vectors of an iteration
// outgrow L2 and the update is bound by HBM (121x181x361 FP64: 73 -> 59 us an
// iteration; 127x181x361 refined: 52 -> 41); below that x stays in L2 and a
// launch per group costs more than it saves (63x91x181: 11.1 -> 12.9 us).
// The buffers are vectors that the handle has anyway and that an inner
// iteration leaves alone, so a rotation takes no memory: d_tmp and the staging
// of host vectors (FP64), the halves of d_p, d_p2 and d_tmp (refined).  Every
// valid point of a direction is written before it is read; pad lanes may hold
// anything, no result depends on them.
int Solver::x_buffers() {
  if (batched) return POT3D_OK;  // batches update x in pairs from the two buffers
  int dev = 0, l2 = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
  if (precision == POT3D_FP64) {
    // x, r, p, p', q and a_i against L2; on grids of fewer than eight radial
    // points the padded vector can be longer than the staging
    if (ifprec == 2 || 44LL * g.Np <= l2 || 2 * g.N < g.Np) return POT3D_OK;
    double *const q[X_GROUP64] = {d_p, d_p2, d_tmp, d_io};
    std::copy(q, q + X_GROUP64, m_p64q);
    xg64 = X_GROUP64;
    return POT3D_OK;
  }
  float *const h[3] = {reinterpret_cast<float *>(d_p), reinterpret_cast<float *>(d_p2), reinterpret_cast<float *>(d_tmp)};
  float *const q[X_GROUP] = {m_p32a, m_p32b, h[0], h[0] + g.Np, h[1], h[1] + g.Np, h[2], h[2] + g.Np};
  std::copy(q, q + X_GROUP, m_p32q);
  if (ifprec == 2 || 28LL * g.Np > l2) xg = X_GROUP;  // x and FP32 r, p, p', q, a_i
  return POT3D_OK;
}

// x += the group's alpha p, the direction of iteration slot i in buffer i + 1
// of the rotation (modulo its length).
template <typename T, int G>
int Solver::launch_x_group(T *const (&dirs)[G]) {
  XDirs<T, G> x;
  for (int i = 0; i < G; i++) x.p[i] = dirs[(i + 1) % G];
  if (ifprec != 2)
    return pot3d_cuda_status(launch_pdl(k_update_x_group<T, G>, dim3(xblocks), dim3(NTHR), 0, stream, g,
                                        (const SolveState *)d_state, d_x, x), "k_update_x_group");
  k_update_x_group<T, G><<<xblocks, NTHR, 0, stream>>>(g, d_state, d_x, x);
  return pot3d_cuda_status(cudaGetLastError(), "k_update_x_group");
}

// One PCG iteration (src/pot3d.F90:4336-4365) at position u of a captured graph.
int Solver::launch_iteration(int u) {
  dim3 grid(g.nit, g.njt, g.nkc);
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  if (xg64 > 1) {  // the rotation: position u reads buffer u % xg64, writes the next
    p_cur = m_p64q[u % xg64];
    p_nxt = m_p64q[(u + 1) % xg64];
  }
  StencilArgs sa{};
  sa.p_old = p_cur;
  sa.p_new = p_nxt;  // ping-pong: neighbouring tiles still read p_old halos
  sa.r = d_r;
  sa.ai = d_ai;
  sa.q = d_q;
  sa.s1z_part = d_s1z;
  sa.s1p = d_s1p;
  sa.st = d_state;
  sa.partials = d_partials;
  UpdateArgs ua{};
  ua.x = d_x;
  ua.p = p_nxt;
  ua.r = d_r;
  ua.q = d_q;
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  StencilMaps mp;
  int stm;
  if ((stm = tensor_map(p_cur, true, &mp.m64[0]))) return stm;
  if (ifprec == 2) {
    sa.z32 = dilu_z32(this);
    mp.m64[1] = mp.m64[0];
    if ((stm = tensor_map(sa.z32, false, &mp.m32[0]))) return stm;
    k_stencil<MODE_PCGZ><<<grid, NTHR, StageLayout<MODE_PCGZ>::smem, stream>>>(mp, g, m, sa);
    ua.r32 = dilu_r32(this);
    k_update_r32<<<grid1d(g.Np / 2), NTHR, 0, stream>>>(g, ua);
    int st = dilu_sweeps(this, true);
    if (st) return st;
    ua.z32 = dilu_z32(this);
    k_update<UPD_ZDOT, true, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  } else {
    if ((stm = tensor_map(d_r, true, &mp.m64[1]))) return stm;
    if ((stm = tensor_map(d_ai, false, &mp.m32[0]))) return stm;
    if (xg64 > 1) sa.xslot1 = 1 + u % xg64;
    CK(launch_pdl(k_stencil<MODE_PCG>, grid, dim3(NTHR), StageLayout<MODE_PCG>::smem, stream, mp, g, m, sa));
    CK(launch_pdl(xg64 > 1 ? k_update<UPD_ITER, false, false, false> : k_update<UPD_ITER, false, false, true>, gridu,
                  dim3(NTHR), 0, stream, g, m, ua));
    int st;
    if (xg64 > 1 && u % xg64 == xg64 - 1 && (st = launch_x_group(m_p64q))) return st;
  }
  std::swap(p_cur, p_nxt);
  return pot3d_cuda_status(cudaGetLastError(), "launch_iteration");
}

// FP64 PCG (cgsolve, src/pot3d.F90:4231-4369) on d_x (guess) and d_b (RHS).
int Solver::cgsolve_padded(bool zero_guess, int ncgmax, double epscg, int *ierr, pot3d_solve_info_t *info) {
  dim3 grid(g.nit, g.njt, g.nkc);
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  int st;
  SolveState s0{};
  s0.epscg = epscg;
  s0.ncgmax = ncgmax;
  s0.hist = d_hist;
  s0.hist_cap = hist_cap;
  CK(cudaMemcpyAsync(d_state, &s0, sizeof(SolveState), cudaMemcpyHostToDevice, stream));
  CK(cudaEventRecord(ev0, stream));
  launches = 0;
  p_cur = d_p;
  p_nxt = d_p2;
  CK(cudaMemsetAsync(p_cur, 0, sizeof(double) * g.Np, stream));
  CK(cudaMemsetAsync(d_s1p, 0, sizeof(double) * 2 * g.NRP, stream));
  CK(cudaMemcpyAsync(d_r, d_b, sizeof(double) * g.Np, cudaMemcpyDeviceToDevice, stream));
  UpdateArgs ua{};
  ua.x = d_x;
  ua.p = p_cur;
  ua.r = d_r;
  ua.q = d_q;
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  // bdotb = b . M^-1 b  (src/pot3d.F90:4293-4298)
  if (ifprec == 2) {
    if ((st = dilu_reset(this))) return st;
    k_cast_r32<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_r, dilu_r32(this));
    if ((st = dilu_sweeps(this, false))) return st;
    ua.z32 = dilu_z32(this);
    k_update<UPD_BDOTB, true><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  } else {
    k_update<UPD_BDOTB, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  }
  launches += (ifprec == 2) ? 2 + sweep_launches() : 1;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  if (h_state->bdotb == 0.0) {  // zero RHS -> zero solution (src/pot3d.F90:4302-4311)
    CK(cudaMemsetAsync(d_x, 0, sizeof(double) * g.Np, stream));
    CK(cudaStreamSynchronize(stream));
    *ierr = 0;
    last_ncg = 0;
    last_epsn = 0.0;
    last_seconds = 0.0;
    if (info) memset(info, 0, sizeof(*info));
    return POT3D_OK;
  }
  // r = b - A x  (src/pot3d.F90:4317-4322)
  if (!zero_guess) {
    if ((st = ax_padded(d_x, d_q))) return st;
    k_axpy_sub<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_q, d_r);
    launches += 3;
  }
  if (ifprec == 2) {
    k_cast_r32<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_r, dilu_r32(this));
    if ((st = dilu_sweeps(this, false))) return st;
    ua.z32 = dilu_z32(this);
    k_update<UPD_INIT, true><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  } else {
    k_update<UPD_INIT, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  }
  launches += (ifprec == 2) ? 2 + sweep_launches() : 1;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  if (h_state->status == ST_RUNNING) {
    // Iterations run in CUDA graphs of 2U iterations; the host polls the
    // device status once per graph while the next graph is already queued.
    const double est_iter_s = (ifprec == 2 ? 140.0 : 90.0) * (double)g.Np / 5.0e12 + 6e-6;
    int U = (int)std::ceil(0.5e-3 / est_iter_s);
    U = std::max(2, std::min(U, 32));
    U += U & 1;  // whole groups of the solution update
    if (!graph_exec || graph_U != U || graph_kind != ifprec) {
      if (graph_exec) cudaGraphExecDestroy(graph_exec);
      graph_exec = nullptr;
      cudaGraph_t graph;
      CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
      for (int u = 0; u < 2 * U; u++) {  // a multiple of 4: the rotation returns to d_p
        st = launch_iteration(u);
        if (st) {
          cudaStreamEndCapture(stream, &graph);
          if (graph) cudaGraphDestroy(graph);
          return st;
        }
      }
      CK(cudaStreamEndCapture(stream, &graph));
      cudaError_t e = cudaGraphInstantiate(&graph_exec, graph, 0);
      cudaGraphDestroy(graph);
      CK(e);
      graph_U = U;
      graph_kind = ifprec;
    }
    const long long per_graph = 2LL * U;
    const long long nodes = per_graph * ((ifprec == 2) ? 3 + sweep_launches() : 2) + (xg64 > 1 ? per_graph / xg64 : 0);
    long long launched = per_graph;
    int last_seen = -1, stalls = 0;
    CK(cudaGraphLaunch(graph_exec, stream));
    launches += nodes;
    for (;;) {
      CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
      CK(cudaEventRecord(ev1, stream));
      if (launched < (long long)ncgmax + per_graph) {
        CK(cudaGraphLaunch(graph_exec, stream));
        launched += per_graph;
        launches += nodes;
      }
      CK(cudaEventSynchronize(ev1));
      if (h_state->status != ST_RUNNING) break;
      if (launched >= (long long)ncgmax + 2 * per_graph) break;
      // A running state must advance by a whole graph per poll.
      if (h_state->ncg <= last_seen) {
        if (++stalls >= 3) {
          pot3d_set_error("PCG state stopped advancing on the device");
          return POT3D_ERR_TIMEOUT;
        }
      } else {
        stalls = 0;
      }
      last_seen = h_state->ncg;
    }
  }
  CK(cudaEventRecord(ev1, stream));
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev0, ev1);
  last_ncg = h_state->ncg;
  last_epsn = h_state->epsn;
  last_seconds = ms * 1e-3;
  last_refine = 0;
  if (h_state->status == ST_BREAKDOWN) {
    pot3d_set_error("PCG breakdown (non-finite or zero p.Ap)");
    return POT3D_ERR_BREAKDOWN;
  }
  if (h_state->status == ST_TIMEOUT) {
    pot3d_set_error("a bounded wait for a TMA tile ran out in the stencil kernel");
    return POT3D_ERR_TIMEOUT;
  }
  *ierr = (h_state->status == ST_CONVERGED) ? 0 : 1;
  if (info) {
    info->ncg = last_ncg;
    info->n_refine = 0;
    info->epsn = last_epsn;
    info->seconds = last_seconds;
    info->true_resid = -1.0;
    info->kernel_launches = launches;
  }
  return POT3D_OK;
}

// Stencil and update kernels of the FP64 diagonal PCG timed one by one, in the
// form the solver iterates with (the grouped x update counts with the update).
int Solver::time_kernels(int reps, double ms[2], double bytes[2]) {
  reps = (reps + xg64 - 1) / xg64 * xg64;  // whole groups
  dim3 grid(g.nit, g.njt, g.nkc);
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  SolveState s0{};
  s0.epscg = 0.0;
  s0.ncgmax = 0x7fffffff;
  CK(cudaMemcpyAsync(d_state, &s0, sizeof(SolveState), cudaMemcpyHostToDevice, stream));
  CK(cudaMemcpyAsync(d_r, d_b, sizeof(double) * g.Np, cudaMemcpyDeviceToDevice, stream));
  CK(cudaMemsetAsync(d_x, 0, sizeof(double) * g.Np, stream));
  CK(cudaMemsetAsync(d_p, 0, sizeof(double) * g.Np, stream));
  CK(cudaMemsetAsync(d_s1p, 0, sizeof(double) * 2 * g.NRP, stream));
  UpdateArgs ua{};
  ua.x = d_x;
  ua.p = d_p;
  ua.r = d_r;
  ua.q = d_q;
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  k_update<UPD_BDOTB, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  k_update<UPD_INIT, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  CK(cudaGetLastError());
  cudaEvent_t e[3];
  for (auto &x : e) CK(cudaEventCreate(&x));
  double t0 = 0, t1 = 0;
  p_cur = d_p;
  p_nxt = d_p2;
  for (int it = 0; it < reps; it++) {
    StencilArgs sa{};
    if (xg64 > 1) {
      p_cur = m_p64q[it % xg64];
      p_nxt = m_p64q[(it + 1) % xg64];
      sa.xslot1 = 1 + it % xg64;
    }
    sa.p_old = p_cur;
    sa.p_new = p_nxt;
    sa.r = d_r;
    sa.ai = d_ai;
    sa.q = d_q;
    sa.s1z_part = d_s1z;
    sa.s1p = d_s1p;
    sa.st = d_state;
    sa.partials = d_partials;
    ua.p = p_nxt;
    StencilMaps mp;
    int stm;
    if ((stm = tensor_map(p_cur, true, &mp.m64[0])) || (stm = tensor_map(d_r, true, &mp.m64[1])) ||
        (stm = tensor_map(d_ai, false, &mp.m32[0])))
      return stm;
    CK(cudaEventRecord(e[0], stream));
    k_stencil<MODE_PCG><<<grid, NTHR, StageLayout<MODE_PCG>::smem, stream>>>(mp, g, m, sa);
    CK(cudaEventRecord(e[1], stream));
    if (xg64 > 1)
      k_update<UPD_ITER, false, false, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    else
      k_update<UPD_ITER, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    if (xg64 > 1 && it % xg64 == xg64 - 1 && (stm = launch_x_group(m_p64q))) return stm;
    CK(cudaEventRecord(e[2], stream));
    CK(cudaEventSynchronize(e[2]));
    float a = 0.f, b = 0.f;
    cudaEventElapsedTime(&a, e[0], e[1]);
    cudaEventElapsedTime(&b, e[1], e[2]);
    t0 += a;
    t1 += b;
    std::swap(p_cur, p_nxt);
  }
  for (auto &x : e) cudaEventDestroy(x);
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  if (h_state->status != ST_RUNNING) {
    pot3d_set_error("kernel timing run left the running state");
    return POT3D_ERR_BREAKDOWN;
  }
  ms[0] = t0 / reps;
  ms[1] = t1 / reps;
  bytes[0] = 32.0 * (double)g.N;
  bytes[1] = (32.0 + 16.0 / xg64) * (double)g.N;
  return POT3D_OK;
}

// ||b - A x||_2 / ||b||_2 of d_x against d_b (d_q, d_tmp as scratch).
int Solver::sweep_launches() const { return ifprec == 2 ? dilu_sweep_launches(const_cast<Solver *>(this)) : 0; }

int Solver::true_residual(double *out) {
  int st;
  if ((st = ax_padded(d_x, d_q))) return st;
  CK(cudaMemcpyAsync(d_tmp, d_b, sizeof(double) * g.Np, cudaMemcpyDeviceToDevice, stream));
  k_axpy_sub<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_q, d_tmp);
  if ((st = dot_padded(d_tmp, d_tmp, d_scalar))) return st;
  if ((st = dot_padded(d_b, d_b, d_scalar + 1))) return st;
  double h[2];
  CK(cudaMemcpyAsync(h, d_scalar, 2 * sizeof(double), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  *out = h[1] > 0 ? std::sqrt(h[0] / h[1]) : 0.0;
  return POT3D_OK;
}

// potfld's phi finalisation, src/pot3d.F90:3966-3969.
int Solver::finalize_phi_dev(const double *xpad, double *phi) {
  const long long n = (long long)g.nr * g.nt * g.np;
  k_phi_interior<<<grid1d(n), NTHR, 0, stream>>>(g, m, xpad, phi);
  k_phi_ring<<<(g.nr + 127) / 128, 128, 0, stream>>>(g, m, phi, d_sums);
  k_phi_poles<<<grid1d((long long)g.nr * (g.np - 2)), NTHR, 0, stream>>>(g, d_sums, phi);
  k_phi_seam<<<grid1d((long long)g.nr * g.nt), NTHR, 0, stream>>>(g, phi);
  return pot3d_cuda_status(cudaGetLastError(), "finalize_phi");
}

int Solver::getb_dev(const double *phi, double *br, double *bt, double *bp) {
  const long long n = (long long)g.nr * g.nt * g.np;
  k_getb<<<grid1d(n), NTHR, 0, stream>>>(g, m, phi, br, bt, bp);
  return pot3d_cuda_status(cudaGetLastError(), "getb");
}

int Solver::energy_dev(const double *phi, double w[3]) {
  const int nb = 148 * 4;
  k_energy<<<nb, NTHR, 0, stream>>>(g, m, phi, d_partials);
  k_energy_final<<<1, 96, 0, stream>>>(d_partials, nb, d_scalar);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(w, d_scalar, 3 * sizeof(double), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  return POT3D_OK;
}

}  // namespace pot3d

namespace pot3d {

float *Solver::r32_inner() { return ifprec == 2 ? dilu_r32(this) : m_r32; }

// One FP32-inner iteration at position u of a captured graph.  Diagonal
// preconditioner: the PCG32 stencil (p = beta p + a_i r, q = A p, p.q ->
// alpha) and the update (x += alpha p, r -= alpha q, r.(a_i r) -> rho,
// beta, epsn).  ILU(0): the PCGZ32 stencil (p = z + beta p), at every
// eighth u the solution update of the last eight iterations, the fused
// sweeps (r32 -= alpha q; r32 -> z32; rho, beta, epsn), the south-ring sums
// of z.
int Solver::launch_iteration32(int u) {
  dim3 grid(g.nit, g.njt, g.nkc);
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  // the rotation: position u reads buffer u % n, writes the next (the two buffers alternate without groups)
  const int nrot = std::max(xg, 2);
  p32_cur = m_p32q[u % nrot];
  p32_nxt = m_p32q[(u + 1) % nrot];
  StencilArgs sa{};
  sa.p_new32 = p32_nxt;
  sa.q32 = m_q32;
  sa.s1z_part = d_s1z;
  sa.s1p = d_s1p;
  sa.st = d_state;
  sa.partials = d_partials;
  sa.xslot1 = xg > 1 ? 1 + u % xg : 0;
  UpdateArgs ua{};
  ua.x = d_x;
  ua.p32 = p32_nxt;
  ua.q32 = m_q32;
  ua.r32 = r32_inner();
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  StencilMaps mp;
  int stm;
  if ((stm = tensor_map(p32_cur, false, &mp.m32[0]))) return stm;
  mp.m64[0] = mp.m64[1] = mp.m32[0];
  if (ifprec == 2) {
    if ((stm = tensor_map(dilu_z32(this), false, &mp.m32[1]))) return stm;
    mp.m32[2] = mp.m32[0];
    k_stencil<MODE_PCGZ32><<<grid, NTHR, StageLayout<MODE_PCGZ32>::smem, stream>>>(mp, g, m, sa);
    // after every eighth iteration x += the eight iterations' alpha p; the
    // sweeps with r32 -= alpha q, rho, beta and ernorm inside them; the
    // south-ring sums of z
    int st;
    if (u % xg == xg - 1 && (st = launch_x_group(m_p32q))) return st;
    if ((st = dilu_sweeps_fused(this, m_q32))) return st;
    k_south_ring_z<<<dim3((g.nrm2 + 127) / 128, g.nkc_u), 128, 0, stream>>>(g, m, (const float *)dilu_z32(this), d_s1z);
  } else {
    if ((stm = tensor_map(m_r32, false, &mp.m32[1])) || (stm = tensor_map(d_ai, false, &mp.m32[2]))) return stm;
    CK(launch_pdl(k_stencil<MODE_PCG32>, grid, dim3(NTHR), StageLayout<MODE_PCG32>::smem, stream, mp, g, m, sa));
    CK(launch_pdl(xg > 1 ? k_update<UPD_ITER, false, true, false> : k_update<UPD_ITER, false, true, true>, gridu,
                  dim3(NTHR), 0, stream, g, m, ua));
    int st;
    if (xg > 1 && u % xg == xg - 1 && (st = launch_x_group(m_p32q))) return st;
  }
  std::swap(p32_cur, p32_nxt);
  return pot3d_cuda_status(cudaGetLastError(), "launch_iteration32");
}

// Reliable update: r = b - A x in FP64 (and its FP32 copy), z = M^-1 r, and
// rho = r.z with the reference's epsn of that residual (UPD_RU).
int Solver::reliable_update() {
  int st;
  if ((st = ax_padded(d_x, d_q))) return st;
  k_resid_cast<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_b, d_q, d_r, r32_inner());
  if (ifprec == 2 && (st = dilu_r_stream(this))) return st;  // the inner iterations' residual
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  UpdateArgs ua{};
  ua.x = d_x;
  ua.r = d_r;
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  if (ifprec == 2) {
    if ((st = dilu_sweeps(this, false))) return st;
    ua.z32 = dilu_z32(this);
    k_update<UPD_RU, true><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    launches += 5 + sweep_launches();
  } else {
    k_update<UPD_RU, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    launches += 4;
  }
  return pot3d_cuda_status(cudaGetLastError(), "reliable_update");
}

// FP32-inner / FP64-refined PCG on d_x (guess) and d_b (RHS), the same
// contract as cgsolve_padded.  Iterations run in CUDA graphs; between graphs
// the host reads the device state and, when the recurrence's rho has fallen
// by refine_ratio since the last reliable update or the recurrence reports
// convergence (or ncgmax), makes a reliable update.  A reliable update whose
// FP64 r.z fell by less than stall_drop is stagnant; stall_limit of them in
// a row hand the solve to the FP64 PCG (cgsolve_padded) from the current x.
int Solver::mixed_solve(bool zero_guess, int ncgmax, double epscg, int *ierr, pot3d_solve_info_t *info) {
  dim3 gridu(g.nit, g.njt, g.nkc_u);
  const bool ilu = ifprec == 2;
  int st;
  SolveState s0{};
  s0.epscg = epscg;
  s0.ncgmax = ncgmax;
  s0.hist = d_hist;
  s0.hist_cap = hist_cap;
  CK(cudaMemcpyAsync(d_state, &s0, sizeof(SolveState), cudaMemcpyHostToDevice, stream));
  CK(cudaEventRecord(evm0, stream));
  launches = 0;
  last_fallback_iters = 0;
  p32_cur = m_p32a;
  p32_nxt = m_p32b;
  CK(cudaMemsetAsync(p32_cur, 0, sizeof(float) * g.Np, stream));  // (m_p32q[0] with ILU(0))
  CK(cudaMemsetAsync(d_s1p, 0, sizeof(double) * 2 * g.NRP, stream));
  CK(cudaMemcpyAsync(d_r, d_b, sizeof(double) * g.Np, cudaMemcpyDeviceToDevice, stream));
  UpdateArgs ua{};
  ua.x = d_x;
  ua.r = d_r;
  ua.ai = d_ai;
  ua.s1z_part = d_s1z;
  ua.st = d_state;
  ua.partials = d_partials;
  // bdotb = b . M^-1 b  (src/pot3d.F90:4293-4298); with ILU(0) this leaves
  // r32 = (float)b and z32 = M^-1 b
  k_cast_r32<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_r, r32_inner());
  launches += 1;
  if (ilu) {
    if ((st = dilu_r_stream(this))) return st;  // the inner iterations' residual (zero guess)
    launches += 1;
    if ((st = dilu_reset(this))) return st;
    if ((st = dilu_sweeps(this, false))) return st;
    ua.z32 = dilu_z32(this);
    k_update<UPD_BDOTB, true><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    launches += 1 + sweep_launches();
  } else {
    k_update<UPD_BDOTB, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
    launches += 1;
  }
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  if (h_state->bdotb == 0.0) {  // zero RHS -> zero solution (src/pot3d.F90:4302-4311)
    CK(cudaMemsetAsync(d_x, 0, sizeof(double) * g.Np, stream));
    CK(cudaStreamSynchronize(stream));
    *ierr = 0;
    last_ncg = 0;
    last_epsn = 0.0;
    last_seconds = 0.0;
    last_refine = 0;
    if (info) memset(info, 0, sizeof(*info));
    return POT3D_OK;
  }
  // initial residual r = b - A x in FP64, z = M^-1 r, rho (src/pot3d.F90:4317-4330)
  if (!zero_guess) {
    if ((st = ax_padded(d_x, d_q))) return st;
    k_resid_cast<<<grid1d(g.Np), NTHR, 0, stream>>>(g.Np, d_b, d_q, d_r, r32_inner());
    launches += 3;
    if (ilu) {
      if ((st = dilu_r_stream(this))) return st;
      if ((st = dilu_sweeps(this, false))) return st;
      launches += 1 + sweep_launches();
    }
  }
  if (ilu)
    k_update<UPD_INIT, true><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  else
    k_update<UPD_INIT, false><<<gridu, NTHR, 0, stream>>>(g, m, ua);
  launches += 1;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));

  // Graphs of 2U iterations (about 2 ms, at most 16): a reliable update is
  // only made between graphs, and it must come before the recurrence has
  // drifted far from the FP64 residual (small grids converge many decades
  // per graph); the host's poll between graphs leaves the GPU idle for a
  // few microseconds.
  const double est_iter_s = (ilu ? 100.0 : 60.0) * (double)g.Np / 5.0e12 + 6e-6;
  int U = (int)std::ceil(2.0e-3 / est_iter_s);
  U = std::max(1, std::min(U, 8));
  U = (U + X_GROUP / 2 - 1) / (X_GROUP / 2) * (X_GROUP / 2);  // whole groups (the rotation and the x update)
  if (!graph32_exec || graph32_U != U) {
    if (graph32_exec) cudaGraphExecDestroy(graph32_exec);
    graph32_exec = nullptr;
    cudaGraph_t graph;
    CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    for (int u = 0; u < 2 * U; u++) {  // a multiple of 8: the directions return to m_p32a
      st = launch_iteration32(u);
      if (st) {
        cudaStreamEndCapture(stream, &graph);
        if (graph) cudaGraphDestroy(graph);
        return st;
      }
    }
    CK(cudaStreamEndCapture(stream, &graph));
    cudaError_t e = cudaGraphInstantiate(&graph32_exec, graph, 0);
    cudaGraphDestroy(graph);
    CK(e);
    graph32_U = U;
  }
  const long long per_graph = 2LL * U;
  // kernels per iteration (ILU(0): stencil, sweeps, ring sums; plus one x
  // update per eight iterations)
  const long long nodes_per_iter = ilu ? 2 + sweep_launches() : 2;
  const long long extra_per_graph = xg > 1 ? 2LL * U / xg : 0;
  double rho_ref = h_state->rho;  // r.z at the last FP64 residual
  int ncg_ref = 0;                // iterations at the last FP64 residual
  int n_refine = 0, stagnant = 0, stalls = 0;
  bool fallback = false;
  while (h_state->status == ST_RUNNING) {
    const int ncg0 = h_state->ncg;
    CK(cudaGraphLaunch(graph32_exec, stream));
    launches += per_graph * nodes_per_iter + extra_per_graph;
    CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    const int status = h_state->status;
    if (status == ST_BREAKDOWN || status == ST_TIMEOUT) break;
    const int ran = h_state->ncg - ncg0;  // iterations of this graph (odd only if it stopped early)
    if (ran <= 0) {
      if (++stalls >= 3) {
        pot3d_set_error("refined PCG state stopped advancing on the device");
        return POT3D_ERR_TIMEOUT;
      }
      continue;
    }
    stalls = 0;
    // reliable update: convergence or ncgmax reported by the recurrence, its
    // r.z fallen by refine_ratio or grown 100x since the last update (PCG's
    // r.z is not monotone), or 1000 iterations without one
    const bool refresh = status == ST_CONVERGED || status == ST_MAXIT || h_state->rho < refine_ratio * rho_ref ||
                         h_state->rho > 100.0 * rho_ref || h_state->ncg - ncg_ref >= 1000;
    if (!refresh) continue;
    if ((st = reliable_update())) return st;
    n_refine++;
    CK(cudaMemcpyAsync(h_state, d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    if (h_state->status != ST_RUNNING) break;
    const int nrot = std::max(xg, 2);
    if (ran % nrot) {
      // the graph stopped inside the rotation: the newest p is in buffer
      // ran % nrot, the next graph's first iteration reads buffer 0
      CK(cudaMemcpyAsync(m_p32q[0], m_p32q[ran % nrot], sizeof(float) * g.Np, cudaMemcpyDeviceToDevice, stream));
    }
    // progress is judged over at least 10 iterations (updates that follow
    // each other closely near convergence neither count nor reset)
    if (h_state->ncg - ncg_ref >= 10) stagnant = (h_state->rho > stall_drop * rho_ref) ? stagnant + 1 : 0;
    rho_ref = h_state->rho;
    ncg_ref = h_state->ncg;
    if (stagnant >= stall_limit) {
      fallback = true;
      break;
    }
  }
  int ncg_total = h_state->ncg;
  int status = h_state->status;
  double epsn = h_state->epsn;
  if (fallback) {
    // the FP32 recurrence stopped tracking the FP64 residual: plain FP64 PCG
    // (same preconditioner) from the current x
    const long long l0 = launches;
    int ie = 1;
    pot3d_solve_info_t inf2{};
    if ((st = cgsolve_padded(false, std::max(1, ncgmax - ncg_total), epscg, &ie, &inf2))) return st;
    launches = l0 + inf2.kernel_launches;
    last_fallback_iters = std::max(1, inf2.ncg);
    ncg_total += inf2.ncg;
    status = ie == 0 ? ST_CONVERGED : ST_MAXIT;
    epsn = inf2.epsn;
  }
  CK(cudaEventRecord(evm1, stream));
  CK(cudaStreamSynchronize(stream));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, evm0, evm1);
  last_ncg = ncg_total;
  last_epsn = epsn;
  last_seconds = ms * 1e-3;
  last_refine = n_refine;
  if (status == ST_BREAKDOWN) {
    pot3d_set_error("refined PCG breakdown (non-finite or zero curvature)");
    return POT3D_ERR_BREAKDOWN;
  }
  if (status == ST_TIMEOUT) {
    pot3d_set_error("a bounded device wait ran out in the refined PCG");
    return POT3D_ERR_TIMEOUT;
  }
  *ierr = (status == ST_CONVERGED) ? 0 : 1;
  if (info) {
    info->ncg = last_ncg;
    info->n_refine = n_refine;
    info->epsn = last_epsn;
    info->seconds = last_seconds;
    info->true_resid = -1.0;
    info->kernel_launches = launches;
  }
  return POT3D_OK;
}

}  // namespace pot3d

// ============================================================================
// Batched PCG: many independent cases (uneven grids, own Br maps, own outer
// radius) advanced together.  One launch of each tiled kernel covers the
// tiles of every unfinished instance: the flat grid is the concatenation of
// the instances' tile grids and each block finds its instance in a table of
// block offsets; instances carry their own tensor maps, vectors, scalars and
// reduction slots, so every instance converges on its own (blocks of a
// finished instance return at once).  All iterations run from CUDA graphs.
// ============================================================================
namespace pot3d {

struct alignas(64) BatchInst {
  StencilMaps maps[2];  // parity 0: p_old = d_p; parity 1: p_old = d_p2
  StencilArgs sa[2];
  UpdateArgs ua[2];
  Geo g;
  DevMesh m;
  unsigned off_s, off_u, off_r;  // first block of the case in the stencil, update and r32-update grids
  unsigned nb_r;                 // blocks of the case in the r32-update grid
};

enum { BATCH_STENCIL = 0, BATCH_UPDATE = 1, BATCH_R32 = 2 };
__device__ __forceinline__ int batch_find(const BatchInst *__restrict__ in, int n, unsigned blk, int which) {
  int i = 0;
  for (int q = 1; q < n; q++) {
    const unsigned o = which == BATCH_STENCIL ? in[q].off_s : which == BATCH_UPDATE ? in[q].off_u : in[q].off_r;
    if (o <= blk) i = q;
  }
  return i;
}

// MODE_PCG (diagonal preconditioner) or MODE_PCGZ (z from the ILU(0) sweeps),
// and their FP32-inner forms MODE_PCG32 / MODE_PCGZ32.
// Three PCGZ32 blocks an SM (80 registers, 64 bytes spilled) against two (114):
// 234 -> 218 us a launch for 12 grids of 63 to 127 x 91 to 181 x 181 to 361.
template <int MODE>
__global__ void __launch_bounds__(NTHR, MODE == MODE_PCGZ32 ? 3 : 2) k_stencil_batch(const BatchInst *__restrict__ in, int n, int par) {
  const int i = batch_find(in, n, blockIdx.x, BATCH_STENCIL);
  const BatchInst &I = in[i];
  const Geo g = I.g;
  const DevMesh m = I.m;
  const StencilArgs a = I.sa[par];
  const unsigned local = blockIdx.x - I.off_s;
  if (threadIdx.x == 0) {  // the thread that issues the TMA loads
    if (MODE == MODE_PCG || MODE == MODE_PCGZ) tma_acquire_desc(&I.maps[par].m64[0]);
    if (MODE == MODE_PCG) tma_acquire_desc(&I.maps[par].m64[1]);
    tma_acquire_desc(&I.maps[par].m32[0]);
    if (MODE == MODE_PCG32 || MODE == MODE_PCGZ32) tma_acquire_desc(&I.maps[par].m32[1]);
    if (MODE == MODE_PCG32) tma_acquire_desc(&I.maps[par].m32[2]);
  }
  stencil_body<MODE>(I.maps[par], g, m, a, local % g.nit, (local / g.nit) % g.njt, local / (g.nit * g.njt));
}

// UPD_ITER with the diagonal preconditioner, UPD_ZDOT after the ILU(0) sweeps
// (R32: the FP32-inner forms).
template <int KIND, bool ZIN, bool R32 = false>
__global__ void __launch_bounds__(NTHR, 4) k_update_batch(const BatchInst *__restrict__ in, int n, int par) {
  const int i = batch_find(in, n, blockIdx.x, BATCH_UPDATE);
  const BatchInst &I = in[i];
  const Geo &g = I.g;
  const unsigned local = blockIdx.x - I.off_u;
  update_body<KIND, ZIN, R32, KIND == UPD_ITER, 2>(g, I.m, I.ua[par], local % g.nit, (local / g.nit) % g.njt, local / (g.nit * g.njt));
}

__global__ void __launch_bounds__(NTHR) k_update_r32_batch(const BatchInst *__restrict__ in, int n, int par) {
  const int i = batch_find(in, n, blockIdx.x, BATCH_R32);
  const BatchInst &I = in[i];
  const unsigned local = blockIdx.x - I.off_r;
  update_r32_body(I.g, I.ua[par], (long long)local * NTHR + threadIdx.x, (long long)I.nb_r * NTHR);
}
// FP32-inner ILU(0), every running case: the paired solution update after
// an odd graph position (the directions of parity 0 and 1, x_pair_body),
// and the south-ring sums of z after the fused sweeps (k_south_ring_z).
__global__ void __launch_bounds__(NTHR) k_update_x_pair_batch(const BatchInst *__restrict__ in, int n) {
  const int i = batch_find(in, n, blockIdx.x, BATCH_R32);
  const BatchInst &I = in[i];
  const unsigned local = blockIdx.x - I.off_r;
  x_pair_body(I.g, I.ua[1].st, I.ua[1].x, I.ua[0].p32, I.ua[1].p32, (long long)local * NTHR + threadIdx.x,
              (long long)I.nb_r * NTHR);
}
__global__ void __launch_bounds__(NTHR) k_south_ring_z_batch(const BatchInst *__restrict__ in, int n) {
  const int i = batch_find(in, n, blockIdx.x, BATCH_R32);
  const BatchInst &I = in[i];
  const unsigned local = blockIdx.x - I.off_r;
  const int neb = (I.g.nrm2 + NTHR - 1) / NTHR;
  for (int w = (int)local; w < neb * I.g.nkc_u; w += (int)I.nb_r)
    south_ring_z_body(I.g, I.m, I.ua[0].z32, I.ua[0].s1z_part, (w % neb) * NTHR + threadIdx.x, w / neb);
}

struct Batch {
  std::vector<Solver *> inst;
  std::vector<int> act;        // cases in the current table (running ones)
  BatchInst *d_tab = nullptr;  // capacity inst.size()
  std::vector<BatchInst> h_tab;
  unsigned nblk_s = 0, nblk_u = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  SolveState *pin = nullptr;  // pinned copies of the cases' states
  cudaGraphExec_t graph = nullptr;
  std::vector<int> graph_act;  // the table the graph was captured for
  int U = 8;
  int tk = 0;      // stencil planes per block (0 = per-case default)
  int tku = 0;     // update kernels' planes per block (0 = per-case default)
  int ifprec = 1;  // 1: diagonal preconditioner; 2: ILU(0) with batched wavefront sweeps
  int precision = POT3D_FP64;  // or POT3D_FP32_REFINED: FP32-inner iterations, per-case reliable updates
  DiluBatch *wave = nullptr;
  unsigned nblk_r = 0;
  std::vector<double *> guess;  // per case: initial guess (padded, device) or null for zero
  // refined mode, per case: r.z at the last FP64 residual and its iteration,
  // iterations at the start of the last graph, updates made, stagnant updates
  // in a row, and the iterations done before a switch to FP64 PCG
  std::vector<double> rho_ref;
  std::vector<int> ncg_ref, ncg0, n_ref, stagnant, ncg_before_fp64;
  ~Batch() {
    if (graph) cudaGraphExecDestroy(graph);
    dilu_batch_destroy(wave);
    for (Solver *s : inst)  // the cases run on the batch's stream, destroyed below
      if (s && s->stream == stream) s->stream = nullptr;
    for (double *g : guess)
      if (g) cudaFree(g);
    if (d_tab) cudaFree(d_tab);
    if (pin) cudaFreeHost(pin);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    for (Solver *s : inst) delete s;
    if (stream) cudaStreamDestroy(stream);
  }
};

// Apply the planes per block to every case (0 keeps each case's default).
static void batch_set_tk(Batch &B, int tk) {
  for (Solver *sp : B.inst) {
    Solver &s = *sp;
    if (tk > 0) {
      s.g.tk = std::min(tk, std::min(s.g.npm2, MAX_TK));
      s.g.nkc = (s.g.npm2 + s.g.tk - 1) / s.g.tk;
    } else {
      s.g.tk = s.tk_default;
      s.g.nkc = s.nkc_default;
    }
  }
  B.tk = tk;
}

// The same for the update kernels' planes per block (0 = per-case default).
// Their ring partials and reduction slots are sized at creation for any
// value >= 8.
static void batch_set_tku(Batch &B, int tku) {
  for (Solver *sp : B.inst) {
    Solver &s = *sp;
    if (tku > 0) {
      s.g.tk_u = std::min(tku, s.g.npm2);
      s.g.nkc_u = (s.g.npm2 + s.g.tk_u - 1) / s.g.tk_u;
    } else {
      s.g.tk_u = s.tku_default;
      s.g.nkc_u = s.nkcu_default;
    }
  }
  B.tku = tku;
}

// Build and upload the instance table of the cases in B.act.
static int batch_table(Batch &B) {
  B.h_tab.assign(B.act.size(), BatchInst{});
  unsigned os = 0, ou = 0, orr = 0;
  const bool ilu = B.ifprec == 2;
  for (size_t t = 0; t < B.act.size(); t++) {
    Solver &s = *B.inst[B.act[t]];
    BatchInst &I = B.h_tab[t];
    I.g = s.g;
    I.m = s.m;
    for (int par = 0; par < 2; par++) {
      double *pold = par == 0 ? s.d_p : s.d_p2, *pnew = par == 0 ? s.d_p2 : s.d_p;
      StencilArgs &sa = I.sa[par];
      sa = StencilArgs{};
      sa.p_old = pold;
      sa.p_new = pnew;
      sa.r = s.d_r;
      sa.ai = s.d_ai;
      sa.q = s.d_q;
      sa.s1z_part = s.d_s1z;
      sa.s1p = s.d_s1p;
      sa.st = s.d_state;
      sa.partials = s.d_partials;
      UpdateArgs &ua = I.ua[par];
      ua = UpdateArgs{};
      ua.x = s.d_x;
      ua.p = pnew;
      ua.r = s.d_r;
      ua.q = s.d_q;
      ua.ai = s.d_ai;
      ua.s1z_part = s.d_s1z;
      ua.st = s.d_state;
      ua.partials = s.d_partials;
      int st;
      if (B.precision == POT3D_FP32_REFINED) {  // the operands of launch_iteration32
        float *o32 = par == 0 ? s.m_p32a : s.m_p32b, *n32 = par == 0 ? s.m_p32b : s.m_p32a;
        sa.p_new32 = n32;
        if (ilu) sa.xslot1 = 1 + par;  // the paired x update (k_update_x_pair_batch)
        sa.q32 = s.m_q32;
        ua.p32 = n32;
        ua.q32 = s.m_q32;
        ua.r32 = s.r32_inner();
        ua.z32 = ilu ? dilu_z32(&s) : nullptr;
        StencilMaps &mp = I.maps[par];
        if ((st = s.tensor_map(o32, false, &mp.m32[0]))) return st;
        if (ilu) {
          if ((st = s.tensor_map(dilu_z32(&s), false, &mp.m32[1]))) return st;
          mp.m32[2] = mp.m32[0];
        } else if ((st = s.tensor_map(s.m_r32, false, &mp.m32[1])) || (st = s.tensor_map(s.d_ai, false, &mp.m32[2]))) {
          return st;
        }
        mp.m64[0] = mp.m64[1] = mp.m32[0];
        continue;
      }
      if (ilu) {  // the operands of launch_iteration's ifprec=2 branch
        sa.z32 = dilu_z32(&s);
        ua.z32 = dilu_z32(&s);
        ua.r32 = dilu_r32(&s);
        if ((st = s.tensor_map(pold, true, &I.maps[par].m64[0])) ||
            (st = s.tensor_map(sa.z32, false, &I.maps[par].m32[0])))
          return st;
        I.maps[par].m64[1] = I.maps[par].m64[0];
      } else {
        if ((st = s.tensor_map(pold, true, &I.maps[par].m64[0])) ||
            (st = s.tensor_map(s.d_r, true, &I.maps[par].m64[1])) ||
            (st = s.tensor_map(s.d_ai, false, &I.maps[par].m32[0])))
          return st;
      }
      I.maps[par].m32[1] = I.maps[par].m32[2] = I.maps[par].m32[0];
    }
    I.off_s = os;
    I.off_u = ou;
    I.off_r = orr;
    I.nb_r = (unsigned)std::max(1LL, std::min((s.g.Np / 2 + NTHR - 1) / NTHR, 148LL * 4));
    os += (unsigned)s.g.nit * s.g.njt * s.g.nkc;
    ou += (unsigned)s.g.nit * s.g.njt * s.g.nkc_u;
    orr += ilu ? I.nb_r : 0;
  }
  B.nblk_s = os;
  B.nblk_u = ou;
  B.nblk_r = orr;
  if (B.act.empty()) return POT3D_OK;
  return pot3d_cuda_status(
      cudaMemcpyAsync(B.d_tab, B.h_tab.data(), sizeof(BatchInst) * B.act.size(), cudaMemcpyHostToDevice, B.stream),
      "cudaMemcpy(batch table)");
}

static int batch_init(Batch &B, int ncgmax, double epscg) {
  const size_t nc = B.inst.size();
  B.rho_ref.assign(nc, 0.0);
  B.ncg_ref.assign(nc, 0);
  B.ncg0.assign(nc, 0);
  B.n_ref.assign(nc, 0);
  B.stagnant.assign(nc, 0);
  B.ncg_before_fp64.assign(nc, -1);
  for (size_t q = 0; q < nc; q++) {
    Solver &s = *B.inst[q];
    const bool guessed = q < B.guess.size() && B.guess[q];
    SolveState s0{};
    s0.epscg = epscg;
    s0.ncgmax = ncgmax;
    s0.hist = nullptr;
    CK(cudaMemcpyAsync(s.d_state, &s0, sizeof(SolveState), cudaMemcpyHostToDevice, B.stream));
    if (guessed)
      CK(cudaMemcpyAsync(s.d_x, B.guess[q], sizeof(double) * s.g.Np, cudaMemcpyDeviceToDevice, B.stream));
    else
      CK(cudaMemsetAsync(s.d_x, 0, sizeof(double) * s.g.Np, B.stream));
    CK(cudaMemsetAsync(s.d_p, 0, sizeof(double) * s.g.Np, B.stream));
    CK(cudaMemsetAsync(s.d_s1p, 0, sizeof(double) * 2 * s.g.NRP, B.stream));
    CK(cudaMemcpyAsync(s.d_r, s.d_b, sizeof(double) * s.g.Np, cudaMemcpyDeviceToDevice, B.stream));
    dim3 gridu(s.g.nit, s.g.njt, s.g.nkc_u);
    UpdateArgs ua{};
    ua.x = s.d_x;
    ua.p = s.d_p;
    ua.r = s.d_r;
    ua.q = s.d_q;
    ua.ai = s.d_ai;
    ua.s1z_part = s.d_s1z;
    ua.st = s.d_state;
    ua.partials = s.d_partials;
    int st;
    if (B.precision == POT3D_FP32_REFINED) {
      // mixed_solve's prologue: bdotb, the FP64 initial residual of the
      // guess and its r.z, with the case's own (unbatched) kernels
      CK(cudaMemsetAsync(s.m_p32a, 0, sizeof(float) * s.g.Np, B.stream));
      k_cast_r32<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_r, s.r32_inner());
      if (B.ifprec == 2) {
        // the fused sweeps' residual stream (zero guess: r = b)
        if ((st = dilu_r_stream(&s)) || (st = dilu_reset(&s)) || (st = dilu_sweeps(&s, false))) return st;
        ua.z32 = dilu_z32(&s);
        k_update<UPD_BDOTB, true><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      } else {
        k_update<UPD_BDOTB, false><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      }
      if (guessed) {
        if ((st = s.ax_padded(s.d_x, s.d_q))) return st;
        k_resid_cast<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_b, s.d_q, s.d_r, s.r32_inner());
        if (B.ifprec == 2 && ((st = dilu_r_stream(&s)) || (st = dilu_sweeps(&s, false)))) return st;
      }
      if (B.ifprec == 2)
        k_update<UPD_INIT, true><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      else
        k_update<UPD_INIT, false><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      continue;
    }
    if (B.ifprec == 2) {
      // bdotb = b . M^-1 b and the initial z, rho as cgsolve_padded does,
      // with the case's own (unbatched) sweeps
      if ((st = dilu_reset(&s))) return st;
      ua.z32 = dilu_z32(&s);
      k_cast_r32<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_r, dilu_r32(&s));
      if ((st = dilu_sweeps(&s, false))) return st;
      k_update<UPD_BDOTB, true><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      if (guessed) {
        if ((st = s.ax_padded(s.d_x, s.d_q))) return st;
        k_axpy_sub<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_q, s.d_r);
      }
      k_cast_r32<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_r, dilu_r32(&s));
      if ((st = dilu_sweeps(&s, false))) return st;
      k_update<UPD_INIT, true><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
    } else {
      k_update<UPD_BDOTB, false><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
      if (guessed) {
        if ((st = s.ax_padded(s.d_x, s.d_q))) return st;
        k_axpy_sub<<<grid1d(s.g.Np), NTHR, 0, B.stream>>>(s.g.Np, s.d_q, s.d_r);
      }
      k_update<UPD_INIT, false><<<gridu, NTHR, 0, B.stream>>>(s.g, s.m, ua);
    }
  }
  if (B.ifprec == 2) {
    int st;
    if ((st = dilu_batch_reset(B.wave, B.stream))) return st;
  }
  return pot3d_cuda_status(cudaGetLastError(), "batch_init");
}

static void batch_iteration(Batch &B, int par) {
  const int n = (int)B.act.size();
  if (B.precision == POT3D_FP32_REFINED) {  // launch_iteration32's sequence, every running case per launch
    if (B.ifprec == 2) {
      k_stencil_batch<MODE_PCGZ32><<<B.nblk_s, NTHR, StageLayout<MODE_PCGZ32>::smem, B.stream>>>(B.d_tab, n, par);
      if (par == 1) k_update_x_pair_batch<<<B.nblk_r, NTHR, 0, B.stream>>>(B.d_tab, n);
      dilu_batch_sweeps_fused(B.wave, B.stream);
      k_south_ring_z_batch<<<B.nblk_r, NTHR, 0, B.stream>>>(B.d_tab, n);
    } else {
      k_stencil_batch<MODE_PCG32><<<B.nblk_s, NTHR, StageLayout<MODE_PCG32>::smem, B.stream>>>(B.d_tab, n, par);
      k_update_batch<UPD_ITER, false, true><<<B.nblk_u, NTHR, 0, B.stream>>>(B.d_tab, n, par);
    }
    return;
  }
  if (B.ifprec == 2) {  // launch_iteration's ifprec=2 sequence, every running case per launch
    k_stencil_batch<MODE_PCGZ><<<B.nblk_s, NTHR, StageLayout<MODE_PCGZ>::smem, B.stream>>>(B.d_tab, n, par);
    k_update_r32_batch<<<B.nblk_r, NTHR, 0, B.stream>>>(B.d_tab, n, par);
    dilu_batch_sweeps(B.wave, B.stream);
    k_update_batch<UPD_ZDOT, true><<<B.nblk_u, NTHR, 0, B.stream>>>(B.d_tab, n, par);
  } else {
    k_stencil_batch<MODE_PCG><<<B.nblk_s, NTHR, StageLayout<MODE_PCG>::smem, B.stream>>>(B.d_tab, n, par);
    k_update_batch<UPD_ITER, false><<<B.nblk_u, NTHR, 0, B.stream>>>(B.d_tab, n, par);
  }
}
// Kernels per batched iteration (the refined ILU(0) form adds one paired x
// update per two iterations, batch_extra_launches_per_graph).
static int batch_launches_per_iteration(const Batch &B) {
  return B.ifprec == 2 ? (B.precision == POT3D_FP32_REFINED ? 4 : 5) : 2;
}
static int batch_extra_launches_per_graph(const Batch &B) {
  return B.ifprec == 2 && B.precision == POT3D_FP32_REFINED ? B.U : 0;
}

// Capture 2U batched iterations of the current table into B.graph.
static int batch_capture(Batch &B) {
  if (B.graph) cudaGraphExecDestroy(B.graph);
  B.graph = nullptr;
  cudaGraph_t graph = nullptr;
  CK(cudaStreamBeginCapture(B.stream, cudaStreamCaptureModeThreadLocal));
  for (int u = 0; u < 2 * B.U; u++) batch_iteration(B, u & 1);  // even: parity returns to 0
  CK(cudaStreamEndCapture(B.stream, &graph));
  cudaError_t e = cudaGraphInstantiate(&B.graph, graph, 0);
  cudaGraphDestroy(graph);
  CK(e);
  B.graph_act = B.act;
  return POT3D_OK;
}

// Time a few iterations of the batch with the current table (all instances
// running); used by the autotuner.
static int batch_time(Batch &B, int iters, float *ms) {
  int st;
  if ((st = batch_init(B, 0x7fffffff, 0.0))) return st;
  batch_iteration(B, 0);
  batch_iteration(B, 1);
  CK(cudaEventRecord(B.ev0, B.stream));
  for (int it = 0; it < iters; it++) batch_iteration(B, it & 1);
  CK(cudaEventRecord(B.ev1, B.stream));
  CK(cudaEventSynchronize(B.ev1));
  cudaEventElapsedTime(ms, B.ev0, B.ev1);
  return pot3d_cuda_status(cudaGetLastError(), "batch_time");
}

static int batch_poll(Batch &B) {
  for (int q : B.act)
    CK(cudaMemcpyAsync(B.pin + q, B.inst[q]->d_state, sizeof(SolveState), cudaMemcpyDeviceToHost, B.stream));
  return pot3d_cuda_status(cudaStreamSynchronize(B.stream), "batch poll");
}

}  // namespace pot3d

struct pot3d_gpu_batch {
  pot3d::Batch b;
};

extern "C" int pot3d_gpu_batch_create_mode(int n, const pot3d_mesh_t *meshes, const double *const *br0s,
                                           const double *pm_r1s, int tk, int ifprec, int precision,
                                           pot3d_gpu_batch **out) {
  using namespace pot3d;
  if (precision != POT3D_FP64 && precision != POT3D_FP32_REFINED) {
    pot3d_set_error("pot3d_gpu_batch_create: precision must be POT3D_FP64 or POT3D_FP32_REFINED");
    return POT3D_ERR_ARG;
  }
  if (n < 1 || !meshes || !br0s || !pm_r1s || !out) {
    pot3d_set_error("pot3d_gpu_batch_create: invalid arguments");
    return POT3D_ERR_ARG;
  }
  if (tk != 0 && (tk < 8 || tk > MAX_TK)) {
    pot3d_set_error("pot3d_gpu_batch_create: planes per block must be 0 or in [8, 512]");
    return POT3D_ERR_ARG;
  }
  if (ifprec != 1 && ifprec != 2) {
    pot3d_set_error("pot3d_gpu_batch_create: ifprec must be 1 (diagonal) or 2 (ILU(0))");
    return POT3D_ERR_ARG;
  }
  *out = nullptr;
  pot3d_gpu_batch *h = new pot3d_gpu_batch();
  Batch &B = h->b;
  B.ifprec = ifprec;
  B.precision = precision;
  B.guess.assign(n, nullptr);
  int st = pot3d_cuda_status(cudaStreamCreate(&B.stream), "cudaStreamCreate");
  if (!st) st = pot3d_cuda_status(cudaEventCreate(&B.ev0), "cudaEventCreate");
  if (!st) st = pot3d_cuda_status(cudaEventCreate(&B.ev1), "cudaEventCreate");
  if (!st) st = pot3d_cuda_status(cudaMallocHost(&B.pin, sizeof(SolveState) * n), "cudaMallocHost");
  if (!st) st = pot3d_cuda_status(cudaMalloc(&B.d_tab, sizeof(BatchInst) * n), "cudaMalloc(batch table)");
  for (int q = 0; q < n && !st; q++) {
    Solver *s = new Solver();
    B.inst.push_back(s);
    s->batched = true;
    st = s->setup(&meshes[q], br0s[q], nullptr, pm_r1s[q], ifprec, precision);
    if (!st) {
      s->tk_default = s->g.tk;
      s->nkc_default = s->g.nkc;
      s->tku_default = s->g.tk_u;
      s->nkcu_default = s->g.nkc_u;
      // reduction slots and south-ring partials for any planes per block >= 8
      const size_t chunks = (size_t)(s->g.npm2 + 7) / 8;
      const size_t need = (size_t)s->g.nit * s->g.njt * chunks;
      if (need > std::max<size_t>(s->nblk_tiled, 148 * 16 * 3))
        st = s->alloc((void **)&s->d_partials, sizeof(double) * need);
      if (!st && chunks > (size_t)s->g.nkc_u)
        st = s->alloc((void **)&s->d_s1z, sizeof(double) * chunks * s->g.NRP);
    }
  }
  // the cases' setup ran on their own streams; from now on they run on the batch's
  if (!st) st = pot3d_cuda_status(cudaDeviceSynchronize(), "batch setup");
  for (Solver *s : B.inst)
    if (!st && s->stream && s->stream != B.stream) {
      cudaStreamDestroy(s->stream);
      s->stream = B.stream;
    }
  if (!st)
    st = pot3d_cuda_status(cudaFuncSetAttribute(k_stencil_batch<MODE_PCG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                StageLayout<MODE_PCG>::smem),
                           "cudaFuncSetAttribute(k_stencil_batch)");
  if (!st)
    st = pot3d_cuda_status(cudaFuncSetAttribute(k_stencil_batch<MODE_PCGZ>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                StageLayout<MODE_PCGZ>::smem),
                           "cudaFuncSetAttribute(k_stencil_batch)");
  for (int m : {MODE_PCG32, MODE_PCGZ32}) {
    if (st) break;
    const void *fn = m == MODE_PCG32 ? (const void *)k_stencil_batch<MODE_PCG32> : (const void *)k_stencil_batch<MODE_PCGZ32>;
    const int smem = m == MODE_PCG32 ? StageLayout<MODE_PCG32>::smem : StageLayout<MODE_PCGZ32>::smem;
    st = pot3d_cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                           "cudaFuncSetAttribute(k_stencil_batch)");
  }
  if (!st && ifprec == 2) st = dilu_batch_setup(B.inst.data(), n, B.stream, &B.wave);
  if (st) {
    delete h;
    return st;
  }
  batch_set_tk(B, tk);
  *out = h;
  return POT3D_OK;
}

extern "C" int pot3d_gpu_batch_create_ex(int n, const pot3d_mesh_t *meshes, const double *const *br0s,
                                         const double *pm_r1s, int tk, int ifprec, pot3d_gpu_batch **out) {
  return pot3d_gpu_batch_create_mode(n, meshes, br0s, pm_r1s, tk, ifprec, POT3D_FP64, out);
}

extern "C" int pot3d_gpu_batch_create(int n, const pot3d_mesh_t *meshes, const double *const *br0s,
                                      const double *pm_r1s, int tk, pot3d_gpu_batch **out) {
  return pot3d_gpu_batch_create_mode(n, meshes, br0s, pm_r1s, tk, 1, POT3D_FP64, out);
}

extern "C" int pot3d_gpu_batch_set_guess(pot3d_gpu_batch *h, int i, const double *x) {
  using namespace pot3d;
  if (!h || i < 0 || i >= (int)h->b.inst.size()) {
    pot3d_set_error("pot3d_gpu_batch_set_guess: invalid arguments");
    return POT3D_ERR_ARG;
  }
  Batch &B = h->b;
  Solver &s = *B.inst[i];
  if (!x) {  // back to a zero guess
    if (B.guess[i]) cudaFree(B.guess[i]);
    B.guess[i] = nullptr;
    return POT3D_OK;
  }
  if (!B.guess[i]) CK(cudaMalloc(&B.guess[i], sizeof(double) * s.g.Np));
  int st;
  CK(cudaMemcpyAsync(s.d_tmp, x, sizeof(double) * s.g.N, cudaMemcpyHostToDevice, B.stream));
  if ((st = s.pack(s.d_tmp, B.guess[i]))) return st;
  CK(cudaStreamSynchronize(B.stream));
  return POT3D_OK;
}

// Autotuner: times `iters` batched iterations of all cases for each candidate
// planes per block; applies and returns the fastest.
extern "C" int pot3d_gpu_batch_tune2(pot3d_gpu_batch *h, const int *cand_tk, int n_tk, const int *cand_tku, int n_tku,
                                     int iters, int *best_tk, int *best_tku, float *ms_out) {
  using namespace pot3d;
  if (!h || !cand_tk || n_tk < 1 || !cand_tku || n_tku < 1 || iters < 1) {
    pot3d_set_error("pot3d_gpu_batch_tune2: invalid arguments");
    return POT3D_ERR_ARG;
  }
  Batch &B = h->b;
  for (int c = 0; c < n_tk; c++)
    if (cand_tk[c] < 8 || cand_tk[c] > MAX_TK) {
      pot3d_set_error("pot3d_gpu_batch_tune2: stencil planes per block must be in [8, 512]");
      return POT3D_ERR_ARG;
    }
  for (int c = 0; c < n_tku; c++)
    if (cand_tku[c] < 8) {
      pot3d_set_error("pot3d_gpu_batch_tune2: update planes per block must be at least 8");
      return POT3D_ERR_ARG;
    }
  float best = 1e30f;
  int bt = cand_tk[0], btu = cand_tku[0], st;
  B.act.resize(B.inst.size());
  for (size_t q = 0; q < B.inst.size(); q++) B.act[q] = (int)q;
  for (int c = 0; c < n_tk; c++)
    for (int d = 0; d < n_tku; d++) {
      batch_set_tk(B, cand_tk[c]);
      batch_set_tku(B, cand_tku[d]);
      if ((st = batch_table(B))) return st;
      float ms = 0.f;
      if ((st = batch_time(B, iters, &ms))) return st;
      if (ms_out) ms_out[c * n_tku + d] = ms;
      if (ms < best) {
        best = ms;
        bt = cand_tk[c];
        btu = cand_tku[d];
      }
    }
  batch_set_tk(B, bt);
  batch_set_tku(B, btu);
  B.graph_act.clear();  // the graph (if any) belongs to another tiling
  if (best_tk) *best_tk = bt;
  if (best_tku) *best_tku = btu;
  return POT3D_OK;
}

extern "C" int pot3d_gpu_batch_tune(pot3d_gpu_batch *h, const int *candidates, int ncand, int iters, int *best_tk,
                                    float *ms_out) {
  using namespace pot3d;
  if (!h || !candidates || ncand < 1 || iters < 1) {
    pot3d_set_error("pot3d_gpu_batch_tune: invalid arguments");
    return POT3D_ERR_ARG;
  }
  Batch &B = h->b;
  for (int c = 0; c < ncand; c++)
    if (candidates[c] < 8 || candidates[c] > MAX_TK) {
      pot3d_set_error("pot3d_gpu_batch_tune: planes per block must be in [8, 512]");
      return POT3D_ERR_ARG;
    }
  float best = 1e30f;
  int bt = candidates[0], st;
  B.act.resize(B.inst.size());
  for (size_t q = 0; q < B.inst.size(); q++) B.act[q] = (int)q;
  for (int c = 0; c < ncand; c++) {
    batch_set_tk(B, candidates[c]);
    if ((st = batch_table(B))) return st;
    float ms = 0.f;
    if ((st = batch_time(B, iters, &ms))) return st;
    if (ms_out) ms_out[c] = ms;
    if (ms < best) {
      best = ms;
      bt = candidates[c];
    }
  }
  batch_set_tk(B, bt);
  B.graph_act.clear();  // the graph (if any) belongs to another tiling
  if (best_tk) *best_tk = bt;
  return POT3D_OK;
}

extern "C" int pot3d_gpu_batch_solve(pot3d_gpu_batch *h, int ncgmax, double epscg, int *ierr,
                                     pot3d_solve_info_t *info, double *seconds) {
  using namespace pot3d;
  if (!h) {
    pot3d_set_error("null batch");
    return POT3D_ERR_ARG;
  }
  Batch &B = h->b;
  const int n = (int)B.inst.size();
  int st;
  CK(cudaEventRecord(B.ev0, B.stream));
  if ((st = batch_init(B, ncgmax, epscg))) return st;
  B.act.resize(n);
  for (int q = 0; q < n; q++) B.act[q] = q;
  if ((st = batch_poll(B))) return st;
  long long launches = 2LL * n;
  // Zero right-hand side -> zero solution (src/pot3d.F90:4302-4311).
  for (int q = 0; q < n; q++)
    if (B.pin[q].bdotb == 0.0) {
      B.pin[q].status = ST_CONVERGED;
      B.pin[q].ncg = 0;
      B.pin[q].epsn = 0.0;
      CK(cudaMemcpyAsync(B.inst[q]->d_state, &B.pin[q], sizeof(SolveState), cudaMemcpyHostToDevice, B.stream));
    }
  // Loop: run 2U iterations of the running cases from a graph, read their
  // states, drop the finished ones from the table (so later launches cover
  // only running cases' tiles) and re-capture when the set changed.
  long long last_total = -1;
  int stalls = 0;
  const bool refined = B.precision == POT3D_FP32_REFINED;
  for (int q = 0; q < n; q++) B.rho_ref[q] = B.pin[q].rho;
  bool after_graph = false;
  for (;;) {
    if (refined && after_graph) {
      // Reliable updates of the cases that need one (mixed_solve's rules,
      // per case), made with each case's own kernels, then one poll.
      std::vector<int> ru;
      for (int q : B.act) {
        const SolveState &S = B.pin[q];
        if (S.status != ST_RUNNING && S.status != ST_CONVERGED && S.status != ST_MAXIT) continue;
        if (B.ncg_before_fp64[q] >= 0) continue;  // finished by FP64 PCG
        if (S.status == ST_CONVERGED || S.status == ST_MAXIT || S.rho < B.inst[q]->refine_ratio * B.rho_ref[q] ||
            S.rho > 100.0 * B.rho_ref[q] || S.ncg - B.ncg_ref[q] >= 1000)
          ru.push_back(q);
      }
      if (!ru.empty()) {
        for (int q : ru)
          if ((st = B.inst[q]->reliable_update())) return st;
        std::vector<int> ran(n, 0);
        for (int q : ru) ran[q] = B.pin[q].ncg - B.ncg0[q];
        if ((st = batch_poll(B))) return st;
        for (int q : ru) {
          Solver &s = *B.inst[q];
          const SolveState &S = B.pin[q];
          B.n_ref[q]++;
          if (S.status != ST_RUNNING) continue;
          if (ran[q] & 1)  // stopped after an odd number of iterations: newest p in the other buffer
            CK(cudaMemcpyAsync(s.m_p32a, s.m_p32b, sizeof(float) * s.g.Np, cudaMemcpyDeviceToDevice, B.stream));
          if (S.ncg - B.ncg_ref[q] >= 10) B.stagnant[q] = S.rho > s.stall_drop * B.rho_ref[q] ? B.stagnant[q] + 1 : 0;
          B.rho_ref[q] = S.rho;
          B.ncg_ref[q] = S.ncg;
          if (B.stagnant[q] >= s.stall_limit) {
            // this case's FP32 recurrence stopped tracking its FP64 residual:
            // FP64 PCG (same preconditioner) from its current x, on its own
            B.ncg_before_fp64[q] = S.ncg;
            int ie = 1;
            pot3d_solve_info_t inf2{};
            if ((st = s.cgsolve_padded(false, std::max(1, ncgmax - S.ncg), epscg, &ie, &inf2))) return st;
          }
        }
        if ((st = batch_poll(B))) return st;
      }
    }
    std::vector<int> run;
    long long total = 0;  // iterations of all cases, finished ones included
    for (int q : B.act)
      if (B.pin[q].status == ST_RUNNING) run.push_back(q);
    for (int q = 0; q < n; q++) total += B.pin[q].ncg;
    if (run.empty()) break;
    if (total <= last_total) {
      if (++stalls >= 3) {
        pot3d_set_error("batched PCG state stopped advancing on the device");
        return POT3D_ERR_TIMEOUT;
      }
    } else {
      stalls = 0;
    }
    last_total = total;
    if (run != B.act || !B.graph || B.graph_act != run) {
      B.act = run;
      if ((st = batch_table(B)) || (st = batch_capture(B))) return st;
    }
    for (int q : run) B.ncg0[q] = B.pin[q].ncg;
    CK(cudaGraphLaunch(B.graph, B.stream));
    launches += 2LL * B.U * batch_launches_per_iteration(B) + batch_extra_launches_per_graph(B);
    if ((st = batch_poll(B))) return st;
    after_graph = true;
  }
  CK(cudaEventRecord(B.ev1, B.stream));
  CK(cudaEventSynchronize(B.ev1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, B.ev0, B.ev1);
  for (int q = 0; q < n; q++) {
    if (ierr) ierr[q] = B.pin[q].status == ST_CONVERGED ? 0 : 1;
    if (info) {
      info[q] = pot3d_solve_info_t{};
      info[q].ncg = B.pin[q].ncg + std::max(0, B.ncg_before_fp64[q]);
      info[q].n_refine = refined ? B.n_ref[q] : 0;
      info[q].epsn = B.pin[q].epsn;
      info[q].seconds = ms * 1e-3;
      info[q].kernel_launches = launches;
    }
  }
  for (int q = 0; q < n; q++)
    if (B.pin[q].status == ST_BREAKDOWN || B.pin[q].status == ST_TIMEOUT) {
      const bool bd = B.pin[q].status == ST_BREAKDOWN;
      pot3d_set_error(std::string(bd ? "batched PCG breakdown in case " : "TMA wait timed out in case ") +
                      std::to_string(q));
      return bd ? POT3D_ERR_BREAKDOWN : POT3D_ERR_TIMEOUT;
    }
  if (seconds) *seconds = ms * 1e-3;
  return POT3D_OK;
}

extern "C" int pot3d_gpu_batch_solution(pot3d_gpu_batch *h, int i, double *x) {
  using namespace pot3d;
  if (!h || i < 0 || i >= (int)h->b.inst.size() || !x) {
    pot3d_set_error("pot3d_gpu_batch_solution: invalid arguments");
    return POT3D_ERR_ARG;
  }
  Solver &s = *h->b.inst[i];
  int st;
  if ((st = s.unpack(s.d_x, reinterpret_cast<double *>(s.d_tmp)))) return st;
  CK(cudaStreamSynchronize(s.stream));
  CK(cudaMemcpy(x, s.d_tmp, sizeof(double) * s.g.N, cudaMemcpyDeviceToHost));
  return POT3D_OK;
}

extern "C" int pot3d_gpu_batch_destroy(pot3d_gpu_batch *h) {
  delete h;
  return POT3D_OK;
}
