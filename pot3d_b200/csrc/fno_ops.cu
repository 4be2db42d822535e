// Elementwise, layout and optimiser kernels of the learned warm start (the
// Fourier-style neural operator); its contractions run on pot3d_tc_gemm.
//
//   pot3d_fno_permute  4-D permutation with zero padding / cropping and an
//                      optional add into an FP32 output
//   pot3d_fno_gelu     GELU (tanh form) forward, or its derivative applied to
//                      an incoming gradient
//   pot3d_fno_colsum   deterministic column sums (bias gradients)
//   pot3d_fno_relmse   per-sample relative squared error and its gradient
//   pot3d_fno_adam     Adam step on FP32 master weights with a BF16 copy
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pot3d_learned.h"
#include "fno_math.cuh"
#include "pot3d_internal.cuh"

namespace {

enum { DT_F32 = 0, DT_BF16 = 1 };

__device__ __forceinline__ float ld(const void *p, long long i, int dt) {
  return dt == DT_F32 ? reinterpret_cast<const float *>(p)[i]
                      : __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(p)[i]);
}
__device__ __forceinline__ void st(void *p, long long i, int dt, float v) {
  if (dt == DT_F32)
    reinterpret_cast<float *>(p)[i] = v;
  else
    reinterpret_cast<__nv_bfloat16 *>(p)[i] = __float2bfloat16_rn(v);
}

// f(row, column) for every element of rows x cols.  A warp a row spares a
// division per element, but leaves lanes idle on rows of fewer than 32 columns
// and the chip on few rows: those go element by element (4.2 million values a
// GELU: 32 columns 26 us by rows, 1 column 392 by rows and 30 by elements).
__host__ __device__ inline bool by_elements(long long rows, long long cols) { return cols < 32 || rows < 2048; }
template <typename F>
__device__ __forceinline__ void each_element(long long rows, int cols, F f) {
  const long long n = rows * cols;
  if (!by_elements(rows, cols)) {
    for (long long r = blockIdx.x * 8LL + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8LL)
#pragma unroll 4
      for (int c = threadIdx.x & 31; c < cols; c += 32) f(r, c);
  } else if (n < 1LL << 31) {
    for (unsigned t = blockIdx.x * 256u + threadIdx.x; t < (unsigned)n; t += gridDim.x * 256u) {
      const unsigned r = t / (unsigned)cols;
      f((long long)r, (int)(t - r * (unsigned)cols));
    }
  } else {
    for (long long t = blockIdx.x * 256LL + threadIdx.x; t < n; t += gridDim.x * 256LL) f(t / cols, (int)(t % cols));
  }
}

struct Dims4 {
  long long d[4];
};

// out[o0][o1][o2][o3] = in[i] with i[perm[a]] = o[a]; zero where i is
// outside in's extent.  With add, out (FP32) += value.
struct PermArgs {
  const void *in;
  void *out;
  int in_dt, out_dt, add;
  long long is[4];  // in's stride along each out axis
  long long ie[4];  // in's extent along each out axis
  long long od[4];
};
__device__ __forceinline__ void perm_put(const PermArgs &a, long long t, float v) {
  if (a.add)
    reinterpret_cast<float *>(a.out)[t] += v;
  else
    st(a.out, t, a.out_dt, v);
}
// in's fastest axis is out's: whole rows, a warp a row (one set of divisions
// per row instead of per element).
__global__ void __launch_bounds__(256) k_permute_rows(PermArgs a, long long rows) {
  const int lane = threadIdx.x & 31;
  for (long long r = blockIdx.x * 8LL + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8LL) {
    const long long o01 = r / a.od[2];
    const long long o2 = r % a.od[2], o1 = o01 % a.od[1], o0 = o01 / a.od[1];
    const bool inside = o0 < a.ie[0] && o1 < a.ie[1] && o2 < a.ie[2];
    const long long ib = o0 * a.is[0] + o1 * a.is[1] + o2 * a.is[2];
    for (long long c = lane; c < a.od[3]; c += 32)
      perm_put(a, r * a.od[3] + c, inside && c < a.ie[3] ? ld(a.in, ib + c, a.in_dt) : 0.0f);
  }
}
// The same for FP32 rows stored as BF16 without accumulation (a layer's input
// from its FP32 sums): eight columns a thread, two 16-byte loads and one
// 16-byte store.  Rows, columns and strides that keep these aligned only
// (pot3d_fno_permute); indexes are below 2^31.  47 -> 10.5 us for 32 of 64
// columns at 359 x 719 positions.
__global__ void __launch_bounds__(256) k_permute_rows8(PermArgs a, unsigned n) {
  const unsigned cols = (unsigned)(a.od[3] / 8), n2 = (unsigned)a.od[2], n1 = (unsigned)a.od[1];
  for (unsigned t = blockIdx.x * 256u + threadIdx.x; t < n; t += gridDim.x * 256u) {
    const unsigned r = t / cols, c = (t - r * cols) * 8, o01 = r / n2, o2 = r - o01 * n2, o0 = o01 / n1, o1 = o01 - o0 * n1;
    const bool inside = o0 < a.ie[0] && o1 < a.ie[1] && o2 < a.ie[2];
    const float *in = reinterpret_cast<const float *>(a.in) + o0 * a.is[0] + o1 * a.is[1] + o2 * a.is[2] + c;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 f = inside && c < a.ie[3] ? __ldg(reinterpret_cast<const float4 *>(in)) : z;
    const float4 h = inside && c + 4 < a.ie[3] ? __ldg(reinterpret_cast<const float4 *>(in) + 1) : z;
    __align__(16) __nv_bfloat162 o[4] = {__floats2bfloat162_rn(f.x, f.y), __floats2bfloat162_rn(f.z, f.w),
                                         __floats2bfloat162_rn(h.x, h.y), __floats2bfloat162_rn(h.z, h.w)};
    reinterpret_cast<uint4 *>(a.out)[t] = *reinterpret_cast<const uint4 *>(o);
  }
}
// Any permutation, one element at a time: where rows, or the axes to be turned,
// are too short for the forms around it (pot3d_fno_permute).
__global__ void __launch_bounds__(256) k_permute_any(PermArgs a, long long n) {
  for (long long t = blockIdx.x * 256LL + threadIdx.x; t < n; t += gridDim.x * 256LL) {
    long long r = t / a.od[3];
    const long long o3 = t - r * a.od[3], o2 = r % a.od[2];
    r /= a.od[2];
    const long long o1 = r % a.od[1], o0 = r / a.od[1];
    const bool inside = o0 < a.ie[0] && o1 < a.ie[1] && o2 < a.ie[2] && o3 < a.ie[3];
    perm_put(a, t, inside ? ld(a.in, o0 * a.is[0] + o1 * a.is[1] + o2 * a.is[2] + o3 * a.is[3], a.in_dt) : 0.0f);
  }
}
// in's fastest axis is out axis q < 3: tiles of PT3 x 32 over (3, q) turned
// in shared memory, so both sides move whole lines.  u, v: the other two out
// axes.
constexpr int PT3 = 128;
struct TileArgs {
  const void *in;
  void *out;
  long long is3, isu, isv, osq, osu, osv;  // strides along out axes 3, u, v (in) and q, u, v (out)
  long long ieq, ie3, ieu, iev, odq, od3;  // extents (in's along out axes)
  unsigned n3, nq, nv;                     // tiles along 3 and q; out's extent along v
  int add;
};
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) k_permute_tile(const __grid_constant__ TileArgs a) {
  __shared__ float tile[PT3][33];
  const unsigned bl = blockIdx.x;  // below 2^31
  const unsigned i3 = bl % a.n3, iq = bl / a.n3 % a.nq, uv = bl / a.n3 / a.nq;
  const long long b3 = (long long)i3 * PT3, bq = (long long)iq * 32;
  const long long ov = uv % a.nv, ou = uv / a.nv;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const bool inside = ou < a.ieu && ov < a.iev && bq + x < a.ieq;
  const TI *ib = reinterpret_cast<const TI *>(a.in) + ou * a.isu + ov * a.isv + bq + x;
  TI r[PT3 / 8];
#pragma unroll
  for (int k = 0; k < PT3 / 8; k++) {
    const long long o3 = b3 + y + 8 * k;
    r[k] = inside && o3 < a.ie3 ? ib[o3 * a.is3] : TI(0.0f);
  }
#pragma unroll
  for (int k = 0; k < PT3 / 8; k++) tile[y + 8 * k][x] = (float)r[k];
  __syncthreads();
  const long long ob = ou * a.osu + ov * a.osv + b3 + x;
  TO *out = reinterpret_cast<TO *>(a.out);
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const long long oq = bq + y + 8 * s;
    if (oq >= a.odq) break;
#pragma unroll
    for (int k = 0; k < PT3 / 32; k++) {
      if (b3 + x + 32 * k < a.od3) {
        TO *o = out + ob + oq * a.osq + 32 * k;
        const float val = tile[x + 32 * k][y + 8 * s];
        if (a.add)
          *o = (TO)((float)*o + val);  // FP32 only
        else
          *o = (TO)val;
      }
    }
  }
}
// One Fourier layer's sum and activation: pre[m][c] += spec[b][c][ph][th] for
// m = (b, ph, th), and vout[m][0..63] (BF16) = act(pre[m][c]), zero for c >= W.
// keep: pre's sum is stored (the backward pass needs it).  Bound by HBM and
// L2 traffic (4 W + 2 W + 128 bytes a row), so the spectral term of 64 theta
// points is turned in shared memory and a thread then forms eight channels of
// one row: two 16-byte loads of pre and one 16-byte store (VEC: W a multiple of
// four, pre and vout aligned; else one value at a time).  The W channels and the zeros beyond are
// two loops, so that no lane of a warp idles through the activation.  33.7 ->
// 25.1 us at 359 x 719 positions, W = 32, against one channel a lane.
constexpr int SA_TH = 64;
template <bool VEC>
__global__ void __launch_bounds__(256) k_spec_act(float *__restrict__ pre, const __nv_bfloat16 *__restrict__ spec, int W,
                                                  int nph, int nth, int Pth, int act, int keep,
                                                  __nv_bfloat16 *__restrict__ vout) {
  __shared__ float tile[64][SA_TH + 1];
  const int lane = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int tiles = (nth + SA_TH - 1) / SA_TH, th0 = (int)(blockIdx.x % tiles) * SA_TH;
  const int line = blockIdx.x / tiles, b = line / nph, ph = line % nph;
  const int rows = min(SA_TH, nth - th0), nc = (W + 7) / 8;
  const __nv_bfloat16 *sb = spec + ((long long)b * W * nph + ph) * Pth + th0;
#pragma unroll 8
  for (int c = y; c < W; c += 8)
#pragma unroll
    for (int t = lane; t < SA_TH; t += 32)
      if (t < rows) tile[c][t] = __bfloat162float(sb[(long long)c * nph * Pth + t]);
  __syncthreads();
  const long long m0 = (long long)line * nth + th0;
  for (int i = threadIdx.x; i < rows * nc; i += 256) {
    const int r = i / nc, c0 = (i - r * nc) * 8;
    float *q = pre + (m0 + r) * W + c0;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; k += 4) {
      if (VEC) {
        const float4 f = c0 + k < W ? *reinterpret_cast<const float4 *>(q + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[k] = f.x, v[k + 1] = f.y, v[k + 2] = f.z, v[k + 3] = f.w;
      } else {
#pragma unroll
        for (int h = k; h < k + 4; h++) v[h] = c0 + h < W ? q[h] : 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (c0 + k < W) v[k] += tile[c0 + k][r];
    if (keep) {
#pragma unroll
      for (int k = 0; k < 8; k += 4) {
        if (VEC) {
          if (c0 + k < W) *reinterpret_cast<float4 *>(q + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        } else {
#pragma unroll
          for (int h = k; h < k + 4; h++)
            if (c0 + h < W) q[h] = v[h];
        }
      }
    }
    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const float lo = act && c0 + k < W ? gelu_f(v[k]) : v[k], hi = act && c0 + k + 1 < W ? gelu_f(v[k + 1]) : v[k + 1];
      o[k / 2] = __floats2bfloat162_rn(lo, hi);
    }
    __nv_bfloat16 *vo = vout + (m0 + r) * 64 + c0;
    if (VEC) {
      *reinterpret_cast<uint4 *>(vo) = *reinterpret_cast<const uint4 *>(o);
    } else {
#pragma unroll
      for (int k = 0; k < 8; k += 2) vo[k] = o[k / 2].x, vo[k + 1] = o[k / 2].y;
    }
  }
  const int nz = 8 - nc;
  for (int i = threadIdx.x; i < rows * nz; i += 256) {
    const int r = i / nz, c0 = (nc + i - r * nz) * 8;
    __nv_bfloat16 *vo = vout + (m0 + r) * 64 + c0;
    if (VEC) {
      *reinterpret_cast<uint4 *>(vo) = make_uint4(0, 0, 0, 0);
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++) vo[k] = __float2bfloat16_rn(0.0f);
    }
  }
}

// forward: out[m][c] = gelu(pre[m][c]) for c < C, 0 for C <= c < ldo.
// backward: out[m][c] = grad[m][c] * gelu'(pre[m][c]) (c < C), 0 beyond.
__global__ void __launch_bounds__(256) k_gelu(const float *__restrict__ pre, long long M, int C, int ldp,
                                              const void *__restrict__ grad, int g_dt, int ldg, void *__restrict__ out,
                                              int out_dt, int ldo, int backward) {
  each_element(M, ldo, [&](long long m, int c) {
    float v = 0.0f;
    if (c < C) {
      const float x = pre[m * ldp + c];
      v = backward ? ld(grad, m * ldg + c, g_dt) * gelu_d(x) : gelu_f(x);
    }
    st(out, m * ldo + c, out_dt, v);
  });
}

// out[c] = sum_m in[m][c], c < C: partial sums in a fixed order, 64 blocks of
// 256 chains of rows (chain t of block b takes rows 256 b + t, then every
// 256 * 64th) and a binary tree over a block's chains.  1024 threads take CB
// columns (a lane a column, so a warp reads a line of a row, or 32 / CB rows of
// a few columns) and ROWS chains at once; a thread carries the 256 / ROWS
// chains that the tree's widest levels join.
constexpr int CS_CHAINS = 256;
template <int CB>
__global__ void __launch_bounds__(1024) k_colsum(const float *__restrict__ in, long long M, int C, int ld,
                                                 float *__restrict__ part) {
  constexpr int ROWS = CB >= 4 ? 1024 / CB : CS_CHAINS, NC = CS_CHAINS / ROWS;
  const int lane = threadIdx.x % CB, y = threadIdx.x / CB, c = blockIdx.y * CB + lane;
  float s[NC] = {};
  if (c < C) {
    const float *p = in + c;
    const long long step = gridDim.x * (long long)CS_CHAINS;
    long long m0 = blockIdx.x * (long long)CS_CHAINS + y;
#pragma unroll (16 / NC)
    for (; m0 + ROWS * (NC - 1) < M; m0 += step) {
      float v[NC];
#pragma unroll
      for (int j = 0; j < NC; j++) v[j] = p[(m0 + ROWS * j) * ld];
#pragma unroll
      for (int j = 0; j < NC; j++) s[j] += v[j];
    }
#pragma unroll
    for (int j = 0; j < NC; j++)
      if (m0 + ROWS * j < M) s[j] += p[(m0 + ROWS * j) * ld];
  }
#pragma unroll
  for (int o = NC / 2; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < o; j++) s[j] += s[j + o];
  __shared__ float red[ROWS][CB];
  red[y][lane] = s[0];
  __syncthreads();
  for (int o = ROWS / 2; o > 0; o >>= 1) {
    if (y < o) red[y][lane] += red[y + o][lane];
    __syncthreads();
  }
  if (y == 0 && c < C) part[(long long)c * gridDim.x + blockIdx.x] = red[0][lane];
}
__global__ void k_colsum_final(const float *__restrict__ part, int nb, int C, float *__restrict__ out, int add) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float s = 0.0f;
  for (int b = 0; b < nb; b++) s += part[(long long)c * nb + b];
  out[c] = add ? out[c] + s : s;
}

// Per sample b: loss_b = sum (pred - tgt)^2 / sum tgt^2 over npos x R values;
// grad = 2 (pred - tgt) / sum tgt^2 * scale.  pred rows have ldp >= R.  Large
// samples in three launches: up to RM_BLOCKS partial sums a sample, their total
// in a fixed order, the gradient.  (One block a sample did both passes over a
// sample's 8 million values alone: 38 ms for four 127x181x361 samples, against
// 0.2 ms.)  Small ones, and all of them without a workspace, in one: a block or
// a cluster of eight a sample (relmse_one).  The sample is grid.x, which has no
// limit of 65535.
constexpr int RM_BLOCKS = 256;
constexpr int RM_VALUES = 1024;  // values a block takes at least

// A position's values go to 1 to 32 lanes, as many as they are.
__host__ __device__ inline int lanes_of(int n) { return n > 16 ? 32 : n > 8 ? 16 : n > 4 ? 8 : n > 2 ? 4 : n > 1 ? 2 : 1; }

// Sums of (pred - tgt)^2 and tgt^2 over a block's positions (a thread's are p0,
// p0 + step, ...), in every thread of the block.
template <int NW>
__device__ __forceinline__ float2 relmse_sums(const float *__restrict__ pb, int ldp, const void *__restrict__ tgt,
                                              int t_dt, long long tb, long long npos, int R, long long p0,
                                              long long step) {
  const int L = lanes_of(R), lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float se = 0.0f, st2 = 0.0f;
  auto add = [&](long long p, int c) {
    const float tv = ld(tgt, tb + p * R + c, t_dt);
    const float d = pb[p * ldp + c] - tv;
    se += d * d;
    st2 += tv * tv;
  };
  const int c0 = lane & (L - 1);
  if (R > 32) {
    for (long long p = p0; p < npos; p += step)
      for (int c = c0; c < R; c += 32) add(p, c);
  } else if (c0 < R) {
#pragma unroll 8
    for (long long p = p0; p < npos; p += step) add(p, c0);
  }
  __shared__ float r1[NW], r2[NW];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    se += __shfl_xor_sync(0xffffffffu, se, o);
    st2 += __shfl_xor_sync(0xffffffffu, st2, o);
  }
  if (lane == 0) {
    r1[w] = se;
    r2[w] = st2;
  }
  __syncthreads();
  float a = 0.0f, c = 0.0f;
#pragma unroll
  for (int q = 0; q < NW; q++) {
    a += r1[q];
    c += r2[q];
  }
  return make_float2(a, c);
}
__device__ __forceinline__ void relmse_grad(const float *__restrict__ pb, int ldp, const void *__restrict__ tgt,
                                            int t_dt, long long tb, long long npos, int R, float f,
                                            float *__restrict__ gb, long long p0, long long step) {
  const int c0 = threadIdx.x & (lanes_of(ldp) - 1);
  auto put = [&](long long p, int c) {
    gb[p * ldp + c] = c < R ? f * (pb[p * ldp + c] - ld(tgt, tb + p * R + c, t_dt)) : 0.0f;
  };
  if (ldp > 32) {
    for (long long p = p0; p < npos; p += step)
      for (int c = c0; c < ldp; c += 32) put(p, c);
  } else if (c0 < ldp) {
#pragma unroll 4
    for (long long p = p0; p < npos; p += step) put(p, c0);
  }
}
// The position that a thread of block `blk` of NW warps starts from.
template <int NW>
__device__ __forceinline__ long long first_position(int n, unsigned blk) {
  const int L = lanes_of(n);
  return (long long)blk * (NW * (32 / L)) + threadIdx.x / L;
}

__global__ void __launch_bounds__(256) k_relmse_part(const float *__restrict__ pred, int ldp,
                                                     const void *__restrict__ tgt, int t_dt, long long npos, int R,
                                                     float *__restrict__ part) {
  const int b = blockIdx.x;
  const float2 s = relmse_sums<8>(pred + (long long)b * npos * ldp, ldp, tgt, t_dt, (long long)b * npos * R, npos, R,
                                  first_position<8>(R, blockIdx.y), (long long)gridDim.y * 8 * (32 / lanes_of(R)));
  if (threadIdx.x == 0) *reinterpret_cast<float2 *>(part + 2 * ((long long)b * gridDim.y + blockIdx.y)) = s;
}
// den[b] and loss[b] from the sample's partial sums (one warp a sample).
__global__ void k_relmse_sum(const float *__restrict__ part, int nblk, float *__restrict__ den,
                             float *__restrict__ loss) {
  const int b = blockIdx.x, lane = threadIdx.x;
  const float *pb = part + 2LL * b * nblk;
  float se = 0.0f, st2 = 0.0f;
  for (int q = lane; q < nblk; q += 32) {
    se += pb[2 * q];
    st2 += pb[2 * q + 1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    se += __shfl_xor_sync(0xffffffffu, se, o);
    st2 += __shfl_xor_sync(0xffffffffu, st2, o);
  }
  if (lane == 0) {
    const float d = fmaxf(st2, 1e-30f);
    den[b] = d;
    loss[b] = se / d;
  }
}
__global__ void __launch_bounds__(256) k_relmse_grad(const float *__restrict__ pred, int ldp,
                                                     const void *__restrict__ tgt, int t_dt, long long npos, int R,
                                                     float scale, const float *__restrict__ den,
                                                     float *__restrict__ grad) {
  const int b = blockIdx.x;
  relmse_grad(pred + (long long)b * npos * ldp, ldp, tgt, t_dt, (long long)b * npos * R, npos, R, 2.0f * scale / den[b],
              grad + (long long)b * npos * ldp, first_position<8>(ldp, blockIdx.y),
              (long long)gridDim.y * 8 * (32 / lanes_of(ldp)));
}
// A whole sample, by a block or a cluster: both sums (over the cluster's blocks
// in order, read from their shared memory), the loss and the gradient.
template <int NW>
__global__ void __launch_bounds__(32 * NW) k_relmse_one(const float *__restrict__ pred, int ldp,
                                                        const void *__restrict__ tgt, int t_dt, long long npos, int R,
                                                        float scale, float *__restrict__ grad,
                                                        float *__restrict__ loss) {
  const auto cluster = cooperative_groups::this_cluster();
  const unsigned nc = cluster.num_blocks(), rank = cluster.block_rank();
  const long long b = blockIdx.x / nc;
  const float *pb = pred + b * npos * ldp;
  const long long tb = b * npos * R;
  __shared__ float2 mine;
  float2 s = relmse_sums<NW>(pb, ldp, tgt, t_dt, tb, npos, R, first_position<NW>(R, rank),
                             (long long)nc * NW * (32 / lanes_of(R)));
  if (nc > 1) {
    if (threadIdx.x == 0) mine = s;
    cluster.sync();
    s = make_float2(0.0f, 0.0f);
    for (unsigned q = 0; q < nc; q++) {
      const float2 o = *cluster.map_shared_rank(&mine, q);
      s.x += o.x;
      s.y += o.y;
    }
    cluster.sync();
  }
  const float d = fmaxf(s.y, 1e-30f);
  if (rank == 0 && threadIdx.x == 0) loss[b] = s.x / d;
  relmse_grad(pb, ldp, tgt, t_dt, tb, npos, R, 2.0f * scale / d, grad + b * npos * ldp, first_position<NW>(ldp, rank),
              (long long)nc * NW * (32 / lanes_of(ldp)));
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1, float *__restrict__ m2,
                       __nv_bfloat16 *__restrict__ wb, long long n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const float gt = g[t];
    const float a = b1 * m1[t] + (1.0f - b1) * gt;
    const float v = b2 * m2[t] + (1.0f - b2) * gt * gt;
    m1[t] = a;
    m2[t] = v;
    const float upd = lr * (a / c1) / (sqrtf(v / c2) + eps);
    const float nw = w[t] - upd;
    w[t] = nw;
    if (wb) wb[t] = __float2bfloat16_rn(nw);
  }
}

// x[b][p][0] = br0n[b][p]; x[b][p][1..3] = consts[p][0..2]; other channels 0.
// Eight channels (16 bytes) per thread.
__global__ void k_inputs(const float *__restrict__ br0n, const float *__restrict__ consts, long long B, long long npos,
                         __nv_bfloat16 *__restrict__ x, int aligned) {
  const long long n = B * npos * 8;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if ((t & 7) == 0) {
      const long long bp = t >> 3, p = B == 1 ? bp : bp % npos;
      const __nv_bfloat162 a = __float22bfloat162_rn(make_float2(br0n[bp], consts[p * 3])),
                           b = __float22bfloat162_rn(make_float2(consts[p * 3 + 1], consts[p * 3 + 2]));
      w.x = *reinterpret_cast<const unsigned *>(&a);
      w.y = *reinterpret_cast<const unsigned *>(&b);
    }
    if (aligned) {
      reinterpret_cast<uint4 *>(x)[t] = w;
    } else {
      const unsigned h[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int q = 0; q < 8; q++)
        reinterpret_cast<unsigned short *>(x)[8 * t + q] = (unsigned short)(h[q >> 1] >> (16 * (q & 1)));
    }
  }
}

int grid_for(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148LL * 32) b = 148LL * 32;
  return (int)(b < 1 ? 1 : b);
}
int rows_grid(long long rows, long long cols) { return grid_for(rows * (by_elements(rows, cols) ? cols : 32)); }

}  // namespace

extern "C" int pot3d_fno_permute(const void *in, int in_dt, const long long *in_dims, void *out, int out_dt,
                                 const long long *out_dims, const int *perm, int add, void *stream) {
  Dims4 id, od;
  for (int a = 0; a < 4; a++) {
    id.d[a] = in_dims[a];
    od.d[a] = out_dims[a];
    if (id.d[a] < 1 || od.d[a] < 1 || perm[a] < 0 || perm[a] > 3) {
      pot3d_set_error("pot3d_fno_permute: bad dims or permutation");
      return POT3D_ERR_ARG;
    }
  }
  if (add && out_dt != DT_F32) {
    pot3d_set_error("pot3d_fno_permute: add needs an FP32 output");
    return POT3D_ERR_ARG;
  }
  PermArgs a{in, out, in_dt, out_dt, add, {}, {}, {}};
  long long is[4] = {0, 0, 0, 1};
  for (int x = 2; x >= 0; x--) is[x] = is[x + 1] * id.d[x + 1];
  int q = 3;
  for (int x = 0; x < 4; x++) {
    a.is[x] = is[perm[x]];
    a.ie[x] = id.d[perm[x]];
    a.od[x] = od.d[x];
    if (perm[x] == 3) q = x;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (q == 3) {
    const long long rows = od.d[0] * od.d[1] * od.d[2];
    const long long n8 = rows * (a.od[3] / 8);
    if (in_dt == DT_F32 && out_dt == DT_BF16 && !add && a.od[3] % 8 == 0 && a.ie[3] % 4 == 0 && a.is[0] % 4 == 0 &&
        a.is[1] % 4 == 0 && a.is[2] % 4 == 0 && n8 < (1LL << 30) && ((uintptr_t)in | (uintptr_t)out) % 16 == 0)
      k_permute_rows8<<<grid_for(n8), 256, 0, s>>>(a, (unsigned)n8);
    else if (a.od[3] < 64 || rows < 2048)  // 4.2 million values: 1 column 642 us by rows and 28 by elements, 64 25 and 28
      k_permute_any<<<grid_for(rows * a.od[3]), 256, 0, s>>>(a, rows * a.od[3]);
    else
      k_permute_rows<<<grid_for(rows * 32), 256, 0, s>>>(a, rows);
  } else {
    const int u = q == 0 ? 1 : 0, v = q == 2 ? 1 : 2;
    const long long tq = (od.d[q] + 31) / 32, t3 = (od.d[3] + PT3 - 1) / PT3, nb = tq * t3 * od.d[u] * od.d[v];
    const long long n = od.d[0] * od.d[1] * od.d[2] * od.d[3];
    // A tile takes 3 to 4 ns whatever it holds, an element alone 7 ps: tiles
    // from 1024 of their 4096 elements on average (8.4 million elements, axes 3
    // and q of 128 x 8: 40 us against 55; 64 x 8: 69 against 55; 1 x 1: 24,700
    // against 57).
    if (n < 1024 * nb || nb > 0x7fffffff) {
      k_permute_any<<<grid_for(n), 256, 0, s>>>(a, n);
      return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_permute");
    }
    const long long os[4] = {a.od[1] * a.od[2] * a.od[3], a.od[2] * a.od[3], a.od[3], 1};
    const TileArgs t{in,      out,     a.is[3],        a.is[u],         a.is[v],           os[q],
                     os[u],   os[v],   a.ie[q],        a.ie[3],         a.ie[u],           a.ie[v],
                     a.od[q], a.od[3], (unsigned)t3,   (unsigned)tq,    (unsigned)a.od[v], add};
    const unsigned blocks = (unsigned)nb;
    if (in_dt == DT_F32 && out_dt == DT_F32)
      k_permute_tile<float, float><<<blocks, 256, 0, s>>>(t);
    else if (in_dt == DT_F32)
      k_permute_tile<float, __nv_bfloat16><<<blocks, 256, 0, s>>>(t);
    else if (out_dt == DT_F32)
      k_permute_tile<__nv_bfloat16, float><<<blocks, 256, 0, s>>>(t);
    else
      k_permute_tile<__nv_bfloat16, __nv_bfloat16><<<blocks, 256, 0, s>>>(t);
  }
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_permute");
}

extern "C" int pot3d_fno_spec_act(float *pre, const void *spec, int B, int W, int nph, int nth, int Pth, int act,
                                  int keep, void *vout, void *stream) {
  const long long blocks = (long long)B * nph * ((nth + SA_TH - 1) / SA_TH);
  if (B < 1 || W < 1 || W > 64 || nph < 1 || nth < 1 || Pth < nth || blocks > 0x7fffffff) {
    pot3d_set_error("pot3d_fno_spec_act: bad sizes");
    return POT3D_ERR_ARG;
  }
  const auto kernel = W % 4 == 0 && ((uintptr_t)pre | (uintptr_t)vout) % 16 == 0 ? k_spec_act<true> : k_spec_act<false>;
  kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
      pre, reinterpret_cast<const __nv_bfloat16 *>(spec), W, nph, nth, Pth, act, keep,
      reinterpret_cast<__nv_bfloat16 *>(vout));
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_spec_act");
}

extern "C" int pot3d_fno_gelu(const float *pre, long long M, int C, int ldp, const void *grad, int g_dt, int ldg,
                              void *out, int out_dt, int ldo, int backward, void *stream) {
  if (M < 1 || C < 1 || ldp < C || ldo < C || (backward && (!grad || ldg < C))) {
    pot3d_set_error("pot3d_fno_gelu: bad sizes");
    return POT3D_ERR_ARG;
  }
  k_gelu<<<rows_grid(M, ldo), 256, 0, (cudaStream_t)stream>>>(pre, M, C, ldp, grad, g_dt, ldg, out, out_dt, ldo,
                                                               backward);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_gelu");
}

extern "C" int pot3d_fno_colsum(const float *in, long long M, int C, int ld, float *out, int add, float *scratch,
                                int scratch_len, void *stream) {
  const int nb = 64;
  if (M < 1 || C < 1 || ld < C || scratch_len < nb * C) {
    pot3d_set_error("pot3d_fno_colsum: bad sizes or scratch too small");
    return POT3D_ERR_ARG;
  }
  // 4.2 million values in 1, 2, 5 columns: 80, 49, 31 us with 32 lanes for them
  if (C == 1)
    k_colsum<1><<<nb, CS_CHAINS, 0, (cudaStream_t)stream>>>(in, M, C, ld, scratch);
  else if (C <= 8)
    k_colsum<8><<<nb, 1024, 0, (cudaStream_t)stream>>>(in, M, C, ld, scratch);
  else
    k_colsum<32><<<dim3(nb, (C + 31) / 32), 1024, 0, (cudaStream_t)stream>>>(in, M, C, ld, scratch);
  k_colsum_final<<<(C + 127) / 128, 128, 0, (cudaStream_t)stream>>>(scratch, nb, C, out, add);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_colsum");
}

namespace {
// Partial sums a sample: a block takes RM_VALUES values at least.
int relmse_blocks(long long npos, int R) {
  const long long nb = (npos * R + RM_VALUES - 1) / RM_VALUES;
  return (int)(nb < RM_BLOCKS ? nb : RM_BLOCKS);
}
// More samples than two blocks of 1024 threads an SM: a block of 256 each, all
// of them in flight (512 samples of 8192 values: 41 us with 1024, 24 with 256).
constexpr int RM_MANY = 296;
int relmse_one(const float *pred, int ldp, const void *tgt, int t_dt, int nbatch, long long npos, int R, float scale,
               float *grad, float *loss, cudaStream_t s) {
  if (npos * ldp <= 4 * RM_VALUES || nbatch > RM_MANY) {
    k_relmse_one<8><<<nbatch, 256, 0, s>>>(pred, ldp, tgt, t_dt, npos, R, scale, grad, loss);
    return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_relmse");
  }
  const unsigned nc = npos * ldp <= 32 * RM_VALUES ? 1 : 8;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nbatch * nc);
  cfg.blockDim = dim3(1024);
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = nc;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return pot3d_cuda_status(cudaLaunchKernelEx(&cfg, k_relmse_one<32>, pred, ldp, tgt, t_dt, npos, R, scale, grad, loss),
                           "pot3d_fno_relmse");
}
}  // namespace

extern "C" int pot3d_fno_relmse(const float *pred, int ldp, const void *tgt, int t_dt, int nbatch, long long npos,
                                int R, float scale, float *grad, float *loss, void *stream) {
  if (nbatch < 1 || npos < 1 || R < 1 || ldp < R) {
    pot3d_set_error("pot3d_fno_relmse: bad sizes");
    return POT3D_ERR_ARG;
  }
  return relmse_one(pred, ldp, tgt, t_dt, nbatch, npos, R, scale, grad, loss, (cudaStream_t)stream);
}

extern "C" long long pot3d_fno_relmse_scratch(int nbatch) { return (long long)nbatch * (2 * RM_BLOCKS + 1); }

extern "C" int pot3d_fno_relmse_ws(const float *pred, int ldp, const void *tgt, int t_dt, int nbatch, long long npos,
                                   int R, float scale, float *grad, float *loss, float *ws, void *stream) {
  if (nbatch < 1 || npos < 1 || R < 1 || ldp < R || !ws) {
    pot3d_set_error("pot3d_fno_relmse: bad sizes");
    return POT3D_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int nblk = relmse_blocks(npos, R);
  if (nblk < 8 || nbatch > RM_MANY) return relmse_one(pred, ldp, tgt, t_dt, nbatch, npos, R, scale, grad, loss, s);
  float *part = ws, *den = ws + (size_t)nbatch * 2 * nblk;
  k_relmse_part<<<dim3(nbatch, nblk), 256, 0, s>>>(pred, ldp, tgt, t_dt, npos, R, part);
  k_relmse_sum<<<nbatch, 32, 0, s>>>(part, nblk, den, loss);
  const long long nb = (npos * ldp + RM_VALUES - 1) / RM_VALUES;
  k_relmse_grad<<<dim3(nbatch, (unsigned)(nb < 148 * 16 ? nb : 148 * 16)), 256, 0, s>>>(pred, ldp, tgt, t_dt, npos, R,
                                                                                       scale, den, grad);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_relmse");
}

extern "C" int pot3d_fno_adam(float *w, const float *g, float *m1, float *m2, void *wb, long long n, float lr, float b1,
                              float b2, float eps, int step, void *stream) {
  if (n < 1 || step < 1) {
    pot3d_set_error("pot3d_fno_adam: bad sizes");
    return POT3D_ERR_ARG;
  }
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(w, g, m1, m2, reinterpret_cast<__nv_bfloat16 *>(wb), n, lr, b1,
                                                         b2, eps, c1, c2);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_adam");
}

extern "C" int pot3d_fno_inputs(const float *br0n, const float *consts, long long B, long long npos, void *x,
                                void *stream) {
  if (B < 1 || npos < 1) {
    pot3d_set_error("pot3d_fno_inputs: bad sizes");
    return POT3D_ERR_ARG;
  }
  k_inputs<<<grid_for(B * npos * 8), 256, 0, (cudaStream_t)stream>>>(br0n, consts, B, npos,
                                                                    reinterpret_cast<__nv_bfloat16 *>(x),
                                                                    (reinterpret_cast<uintptr_t>(x) & 15) == 0);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_inputs");
}

namespace {
// x[b][pos * R + i] = sigma[b] * out[b][pos][i], i < R: the network output
// (FP32, Rp channels per position) cropped to the radial levels and scaled
// back to the solver's packed FP64 layout (positions (phi, theta), r fastest).
__global__ void __launch_bounds__(256) k_guess(const float *__restrict__ out, long long B, long long npos, int Rp,
                                               int R, const double *__restrict__ sigma, double *__restrict__ x) {
  each_element(B * npos, R, [&](long long bp, int i) {
    x[bp * R + i] = (double)out[bp * Rp + i] * sigma[B == 1 ? 0 : bp / npos];
  });
}
// The same with the radial levels resampled: the network's Rs levels (those
// of the mesh it was trained on) interpolated linearly onto the solver's R
// levels, level i from source levels idx[i] and idx[i]+1 with weight w[i]
// (outside [0, 1] at the ends: linear extrapolation).
// A warp a position: the levels' indices and weights stay in L1.
// Without the staging a row's values are converted to FP64 twice for every
// output, and conversions issue at a tenth of the FP32 rate; STAGED converts a
// row once into shared memory, a warp a row (182 -> 150 us for 125 -> 253
// levels at 359 x 719 positions): where the outputs need at least the row's
// conversions, for rows of up to 768 values, where eight fit 48 KB.  The whole
// row, its padding too, so that every index that is inside a row stays inside.
template <bool STAGED>
__global__ void __launch_bounds__(256) k_guess_resampled(const float *__restrict__ out, long long B, long long npos,
                                                         int Rp, const int *__restrict__ idx,
                                                         const double *__restrict__ w, int R,
                                                         const double *__restrict__ sigma, double *__restrict__ x) {
  if (!STAGED) {
    each_element(B * npos, R, [&](long long bp, int i) {
      const float *o = out + bp * Rp + idx[i];
      const double lo = (double)o[0], hi = (double)o[1];
      x[bp * R + i] = fma(w[i], hi - lo, lo) * sigma[B == 1 ? 0 : bp / npos];
    });
    return;
  }
  extern __shared__ double row_s[];
  const int lane = threadIdx.x & 31;
  double *row = row_s + (threadIdx.x >> 5) * Rp;
  for (long long bp = blockIdx.x * 8LL + (threadIdx.x >> 5); bp < B * npos; bp += gridDim.x * 8LL) {
    const double sg = sigma[bp / npos];
    const float *o = out + bp * Rp;
#pragma unroll 4
    for (int i = lane; i < Rp; i += 32) row[i] = (double)o[i];
    __syncwarp();
#pragma unroll 4
    for (int i = lane; i < R; i += 32) {
      const int q = idx[i];
      const double lo = row[q], hi = row[q + 1];
      x[bp * R + i] = fma(w[i], hi - lo, lo) * sg;
    }
    __syncwarp();
  }
}
}  // namespace

extern "C" int pot3d_fno_guess_resampled(const float *out, long long B, long long npos, int Rp, int Rs,
                                         const int *idx, const double *w, int R, const double *sigma, double *x,
                                         void *stream) {
  if (B < 1 || npos < 1 || R < 1 || Rs < 2 || Rp < Rs) {
    pot3d_set_error("pot3d_fno_guess_resampled: bad sizes");
    return POT3D_ERR_ARG;
  }
  const size_t smem = 8 * sizeof(double) * (size_t)Rp;  // a row for each of the eight warps
  if (smem <= 48 * 1024 && 2LL * R >= Rp && !by_elements(B * npos, R))
    k_guess_resampled<true><<<grid_for(B * npos * 32), 256, smem, (cudaStream_t)stream>>>(out, B, npos, Rp, idx, w, R,
                                                                                          sigma, x);
  else
    k_guess_resampled<false><<<rows_grid(B * npos, R), 256, 0, (cudaStream_t)stream>>>(out, B, npos, Rp, idx, w, R,
                                                                                      sigma, x);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_guess_resampled");
}

extern "C" int pot3d_fno_guess(const float *out, long long B, long long npos, int Rp, int R, const double *sigma,
                               double *x, void *stream) {
  if (B < 1 || npos < 1 || R < 1 || Rp < R) {
    pot3d_set_error("pot3d_fno_guess: bad sizes");
    return POT3D_ERR_ARG;
  }
  k_guess<<<rows_grid(B * npos, R), 256, 0, (cudaStream_t)stream>>>(out, B, npos, Rp, R, sigma, x);
  return pot3d_cuda_status(cudaGetLastError(), "pot3d_fno_guess");
}
