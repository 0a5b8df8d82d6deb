// stencil.cu -- 7-point sweeps, residuals, inner products and BLAS-1 on
// block-structured fields.
//
// Reference routines restated for the GPU (arithmetic order kept, no
// multiply-add contraction, so results match the reference bit for bit where
// the reference is sequential):
//   jacobi_smoother        SolverTest/blas.f90:452-502
//   calc_ax / calc_r / r2  blas.f90:556-698
//   dot                    blas.f90:379-412 (float: exact products, column sums in
//                          float-float, products outside [2^-100, 2^100) in FP64;
//                          block sums in FP64)
//   axpy/xpay/axpyz/axpbypz blas.f90:242-377
// Decomposition: one CTA per block, or per chunk or part of its planes
// (sweep_chunk, sum_parts); sweeps march each (i,j) column along k.
#include <type_traits>

#include "attr.h"
#include "cells.cuh"
#include "common.cuh"
#include "kernels.h"
#include "stream.cuh"
#include "tile.cuh"

namespace bcmg {


// ---------------------------------------------------------------------------
// Deterministic block reduction of one double per thread (fixed tree order).
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (threadIdx.x < nw) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;  // valid in thread 0
}

// ---------------------------------------------------------------------------
// Sweeps over blocks of any shape and operators of coefficient fields:
//   MODE 0 calc_ax, 1 calc_r, 2 calc_r2 (an FP64 partial sum per CTA, sum_parts), 3
//   jacobi_smoother: x1 = x0 - omega (x0 - r/Ap),
//   r = b - Aw xW - Ae xE - As xS - An xN - Ab xB - At xT.
// CC: per-block constants cf8 (rounded to T, RN(1/Ap) last); else the fields, and
// with RECIP the reciprocals of Ap's (op_recip): without them a sweep divides, and
// a trial product before the division would cost it a sixth (16^3, FP64, 4136
// blocks: 907 us with, 741 without, 646 through reciprocals).
//
// CTA (b, z) takes planes [z zc, (z + 1) zc) of block b, a thread a column at a
// time, the loads of U planes issued before the first of them is used: the
// float sweep with coefficient fields moves 40 bytes a cell and is bound by the
// bytes a thread has in flight (4432 blocks of 16^3: 210 us with one plane's).
// Chunks of planes (sweep_chunk) let a mesh of few blocks fill the chip: 328
// blocks of 24x20x12 leave some SMs three blocks and others two.
template <typename T, bool CC, int MODE, int V>
struct SweepCells {
  T w[V], e[V], s[V], n[V], up[V], bv[V], c[CC ? 1 : V][7], rc[V];
};

template <typename T, bool CC, int MODE, int U, bool RECIP = false>
__global__ void __launch_bounds__(256) sweep_kernel(T* __restrict__ out, const T* __restrict__ x,
                                                    const T* __restrict__ bb, Op<T> op, Geom g,
                                                    T omega, int zc,
                                                    double* __restrict__ partial) {
  __shared__ double red[MODE == 2 ? 256 : 1];
  const int b = blockIdx.x;
  const int64_t base = (int64_t)b * g.bstride;
  const int nx = g.nx, ncol = g.nx * g.ny, sy = g.sy, sz = g.sz;
  const int z0 = blockIdx.y * zc, z1 = min(g.nz, z0 + zc);
  const T* xb = x + base;
  const T* rb = MODE != 0 ? bb + base : nullptr;
  T* ob = MODE != 2 ? out + base : nullptr;
  const T* ra = RECIP ? op.rA0 + base : nullptr;
  T cc[8];
  if (CC) {
#pragma unroll
    for (int q = 0; q < 8; q++) cc[q] = op.cf8[(int64_t)b * 8 + q];
  }
  double acc = 0.0;
  for (int ij = threadIdx.x; ij < ncol; ij += blockDim.x) {
    int o = g.at(ij % nx, ij / nx, z0);
    T xm = xb[o - sz], xc = xb[o];
    auto planes = [&](auto vt) {
      constexpr int V = decltype(vt)::value;
      SweepCells<T, CC, MODE, V> d;
#pragma unroll
      for (int u = 0; u < V; u++) {
        const int q = o + u * sz;
        d.w[u] = xb[q - 1];
        d.e[u] = xb[q + 1];
        d.s[u] = xb[q - sy];
        d.n[u] = xb[q + sy];
        d.up[u] = xb[q + sz];
        if (MODE != 0) d.bv[u] = rb[q];
        if (!CC) {
#pragma unroll
          for (int f = 0; f < 7; f++) d.c[u][f] = op.A[f][base + q];
          if (RECIP) d.rc[u] = ra[q];
        }
      }
#pragma unroll
      for (int u = 0; u < V; u++) {
        const T* c = CC ? cc : d.c[CC ? 0 : u];
        const int q = o + u * sz;
        if (MODE == 0) {
          T a = xmul(c[1], d.w[u]);
          a = xadd(a, xmul(c[2], d.e[u]));
          a = xadd(a, xmul(c[3], d.s[u]));
          a = xadd(a, xmul(c[4], d.n[u]));
          a = xadd(a, xmul(c[5], xm));
          a = xadd(a, xmul(c[6], d.up[u]));
          ob[q] = xadd(a, xmul(c[0], xc));
        } else {
          T r = d.bv[u];
          r = xsub(r, xmul(c[1], d.w[u]));
          r = xsub(r, xmul(c[2], d.e[u]));
          r = xsub(r, xmul(c[3], d.s[u]));
          r = xsub(r, xmul(c[4], d.n[u]));
          r = xsub(r, xmul(c[5], xm));
          r = xsub(r, xmul(c[6], d.up[u]));
          if (MODE == 3) {
            const T xt = CC      ? sweep_div(r, c[0], cc[7])
                         : RECIP ? field_div(r, c[0], d.rc[u])
                                 : xdiv(r, c[0]);
            ob[q] = xsub(xc, xmul(omega, xsub(xc, xt)));
          } else {
            r = xsub(r, xmul(c[0], xc));
            if (MODE == 1) ob[q] = r;
            else acc = __fma_rn((double)r, (double)r, acc);
          }
        }
        xm = xc;
        xc = d.up[u];
      }
      o += V * sz;
    };
    int k = z0;
    for (; k + U <= z1; k += U) planes(std::integral_constant<int, U>{});
    for (; k < z1; k++) planes(std::integral_constant<int, 1>{});
  }
  if (MODE == 2) {
    // one tree in two forms: up to four warps gain nothing from packing their pairs
    double none = 0.0;
    if (blockDim.x <= 128) acc = block_sum(acc, red);
    else kr_block_sums<1>(acc, none, red);
    if (threadIdx.x == 0) partial[b * gridDim.y + blockIdx.y] = acc;
  }
}

template <typename T, int MODE>
static cudaError_t launch_sweep(T* out, const T* x, const T* b, const Op<T>& op, const Geom& g,
                                T omega, double* partial, cudaStream_t st) {
  const int parts = sum_parts(g, sizeof(T));
  const int zc = MODE == 2 ? (g.nz + parts - 1) / parts : sweep_chunk(g);
  const dim3 grid(g.nb, (g.nz + zc - 1) / zc);
  const int nt = column_threads(g);
  // planes a round: two for calc_r in FP32 (1408 blocks of 28^3: 118 us, with four
  // 162; 20^3 42 and 55; 288 blocks 15.0 and 17.2), one for calc_r2 in FP64 with
  // fields (8^3, 288 blocks: 8.6 us, with two 9.3)
  constexpr int UC = sizeof(T) == 4 && MODE != 1 ? 4 : 2;
  constexpr int UF = sizeof(T) == 8 && MODE == 2 ? 1 : 2;
  if (op.cc)
    sweep_kernel<T, true, MODE, UC><<<grid, nt, 0, st>>>(out, x, b, op, g, omega, zc, partial);
  else if (MODE == 3 && sizeof(T) == 8 && op.rA0)
    sweep_kernel<T, false, MODE, UF, MODE == 3 && sizeof(T) == 8>
        <<<grid, nt, 0, st>>>(out, x, b, op, g, omega, zc, partial);
  else
    sweep_kernel<T, false, MODE, UF><<<grid, nt, 0, st>>>(out, x, b, op, g, omega, zc, partial);
  return cudaGetLastError();
}

// RN(1/Ap) of every interior cell, 0 where the two-FMA division does not cover
// Ap (div_pre, cells.cuh): made once for the FP64 sweeps of a run or solve.
// Bound by the FP64 pipe: a reciprocal and an integer test of the exponent (a
// division and two compares took 318 us on 18.2 M cells).
__global__ void __launch_bounds__(256) recip_kernel(double* __restrict__ out,
                                                    const double* __restrict__ a, Geom g, int zc) {
  const int64_t base = (int64_t)blockIdx.x * g.bstride;
  const int ncol = g.nx * g.ny;
  const int z0 = blockIdx.y * zc, z1 = min(g.nz, z0 + zc);
  for (int ij = threadIdx.x; ij < ncol; ij += blockDim.x) {
    int64_t o = base + g.at(ij % g.nx, ij / g.nx, z0);
#pragma unroll 4
    for (int k = z0; k < z1; k++, o += g.sz) {
      const double v = a[o];
      const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
      out[o] = e - (1023u - 60u) < 120u ? __drcp_rn(v) : 0.0;
    }
  }
}

cudaError_t launch_recip(double* out, const double* a, const Geom& g, cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  const int zc = sweep_chunk(g);
  recip_kernel<<<dim3(g.nb, (g.nz + zc - 1) / zc), column_threads(g), 0, st>>>(out, a, g, zc);
  return cudaGetLastError();
}

template <typename T>
static bool cubic_fast(const Op<T>& op, const Geom& g) {
  return cubic_residuals(op.cc && op.cf8, g);
}

// jacobi_smoother on cubic blocks with a per-block constant operator: the
// same arithmetic (coefficients rounded to T, the division of the fused
// sweeps), block edge and ghost width fixed at compile time, and each thread
// walking CPT columns side by side so that their loads overlap.
template <typename T, int N, int VC, int CPT>
__global__ void __launch_bounds__(N * N / CPT, CPT > 1 ? (sizeof(T) == 4 ? 4 : 2) : 1) jacobi_cubic_kernel(
    T* __restrict__ x1, const T* __restrict__ x0, const T* __restrict__ bb,
    const T* __restrict__ cf8, Geom g, T omega) {
  using BL = BrickTile<T, N, VC>;
  constexpr int NT = N * N / CPT, LX = BL::LX, LXY = BL::LXY;
  const int b = blockIdx.x;
  const T* cf = cf8 + (int64_t)b * 8;
  const T c0 = cf[0], c1 = cf[1], c2 = cf[2], c3 = cf[3], c4 = cf[4], c5 = cf[5], c6 = cf[6];
  const T rc0 = cf[7];
  const int64_t base = (int64_t)b * g.bstride;
  int off[CPT];
  T xm[CPT], xc[CPT];
#pragma unroll
  for (int c = 0; c < CPT; c++) {
    const int ij = threadIdx.x + c * NT;
    off[c] = BL::at(ij % N, ij / N, 0);
    xm[c] = x0[base + off[c] - LXY];
    xc[c] = x0[base + off[c]];
  }
#pragma unroll 2
  for (int k = 0; k < N; k++) {
    T w[CPT], e[CPT], s_[CPT], n_[CPT], up[CPT], bv[CPT];
#pragma unroll
    for (int c = 0; c < CPT; c++) {
      const T* q = x0 + base + off[c] + k * LXY;
      w[c] = q[-1];
      e[c] = q[1];
      s_[c] = q[-LX];
      n_[c] = q[LX];
      up[c] = q[LXY];
      bv[c] = bb[base + off[c] + k * LXY];
    }
#pragma unroll
    for (int c = 0; c < CPT; c++) {
      T r = bv[c];
      r = xsub(r, xmul(c1, w[c]));
      r = xsub(r, xmul(c2, e[c]));
      r = xsub(r, xmul(c3, s_[c]));
      r = xsub(r, xmul(c4, n_[c]));
      r = xsub(r, xmul(c5, xm[c]));
      r = xsub(r, xmul(c6, up[c]));
      const T xt = sweep_div(r, c0, rc0);
      x1[base + off[c] + k * LXY] = xsub(xc[c], xmul(omega, xsub(xc[c], xt)));
      xm[c] = xc[c];
      xc[c] = up[c];
    }
  }
}

template <typename T>
cudaError_t launch_jacobi(T* x1, const T* x0, const T* b, Op<T> op, const Geom& g, T omega,
                          cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  if (cubic_fast(op, g)) {
    switch (g.nx * 4 + g.vc) {
      case 8 * 4 + 1: jacobi_cubic_kernel<T, 8, 1, 1><<<g.nb, 64, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
      case 8 * 4 + 2: jacobi_cubic_kernel<T, 8, 2, 1><<<g.nb, 64, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
      case 16 * 4 + 1: jacobi_cubic_kernel<T, 16, 1, 1><<<g.nb, 256, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
      case 16 * 4 + 2: jacobi_cubic_kernel<T, 16, 2, 1><<<g.nb, 256, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
      case 32 * 4 + 1: jacobi_cubic_kernel<T, 32, 1, 4><<<g.nb, 256, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
      default: jacobi_cubic_kernel<T, 32, 2, 4><<<g.nb, 256, 0, st>>>(x1, x0, b, op.cf8, g, omega); break;
    }
    return cudaGetLastError();
  }
  return launch_sweep<T, 3>(x1, x0, b, op, g, omega, nullptr, st);
}

// calc_ax / calc_r / calc_r2 on cubic blocks with a constant operator: one
// thread per column, unrolled k walk, coefficients rounded to T on the host;
// calc_r2's block sum in float-float (SqAcc) for float fields.
template <typename T, int N, int VC, int MODE>
__global__ void __launch_bounds__(N * N) residual_cubic_kernel(T* __restrict__ out,
                                                               const T* __restrict__ x,
                                                               const T* __restrict__ bb,
                                                               const T* __restrict__ cf8, Geom g,
                                                               double* __restrict__ partial) {
  using BL = BrickTile<T, N, VC>;
  constexpr int NW = N * N / 32;
  __shared__ double red[NW > 0 ? NW : 1];
  const int b = blockIdx.x, i = threadIdx.x % N, j = threadIdx.x / N;
  const T* cf = cf8 + (int64_t)b * 8;
  const T c0 = cf[0], c1 = cf[1], c2 = cf[2], c3 = cf[3], c4 = cf[4], c5 = cf[5], c6 = cf[6];
  const int64_t p0 = (int64_t)b * g.bstride + BL::at(i, j, 0);
  const T* q = x + p0;
  SqAcc<T> acc;
  T xm = q[-BL::LXY], xc = q[0];
#pragma unroll
  for (int k = 0; k < N; k++) {
    const T* qk = q + k * BL::LXY;
    const T xp = qk[BL::LXY];
    if (MODE == 0) {
      T a = xmul(c1, qk[-1]);
      a = xadd(a, xmul(c2, qk[1]));
      a = xadd(a, xmul(c3, qk[-BL::LX]));
      a = xadd(a, xmul(c4, qk[BL::LX]));
      a = xadd(a, xmul(c5, xm));
      a = xadd(a, xmul(c6, xp));
      a = xadd(a, xmul(c0, xc));
      out[p0 + k * BL::LXY] = a;
    } else {
      T r = bb[p0 + k * BL::LXY];
      r = xsub(r, xmul(c1, qk[-1]));
      r = xsub(r, xmul(c2, qk[1]));
      r = xsub(r, xmul(c3, qk[-BL::LX]));
      r = xsub(r, xmul(c4, qk[BL::LX]));
      r = xsub(r, xmul(c5, xm));
      r = xsub(r, xmul(c6, xp));
      r = xsub(r, xmul(c0, xc));
      if (MODE == 1) out[p0 + k * BL::LXY] = r;
      else acc.add(r);
    }
    xm = xc;
    xc = xp;
  }
  if (MODE == 2) {
    acc.warp_reduce();
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[w] = acc.value();
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = 0.0;
      for (int q2 = 0; q2 < NW; q2++) v += red[q2];
      partial[b] = v;
    }
  }
}

template <typename T, int MODE>
static void residual_cubic(T* out, const T* x, const T* b, const Op<T>& op, const Geom& g,
                           double* partial, cudaStream_t st) {
  const int key = g.nx * 4 + g.vc;
  switch (key) {
    case 8 * 4 + 1: residual_cubic_kernel<T, 8, 1, MODE><<<g.nb, 64, 0, st>>>(out, x, b, op.cf8, g, partial); break;
    case 8 * 4 + 2: residual_cubic_kernel<T, 8, 2, MODE><<<g.nb, 64, 0, st>>>(out, x, b, op.cf8, g, partial); break;
    case 16 * 4 + 1: residual_cubic_kernel<T, 16, 1, MODE><<<g.nb, 256, 0, st>>>(out, x, b, op.cf8, g, partial); break;
    case 16 * 4 + 2: residual_cubic_kernel<T, 16, 2, MODE><<<g.nb, 256, 0, st>>>(out, x, b, op.cf8, g, partial); break;
    case 32 * 4 + 1: residual_cubic_kernel<T, 32, 1, MODE><<<g.nb, 1024, 0, st>>>(out, x, b, op.cf8, g, partial); break;
    default: residual_cubic_kernel<T, 32, 2, MODE><<<g.nb, 1024, 0, st>>>(out, x, b, op.cf8, g, partial); break;
  }
}

// calc_ax / calc_r / calc_r2 of FP64 fields on 16^3 / 32^3 blocks with a constant
// operator: planes streamed through shared memory, each product formed once where
// the six neighbours have one coefficient (stream.cuh).  CTA (b, y): planes [y zc,
// + zc) of block b; calc_r2's partial sum at partial[b * gridDim.y + y].  One
// thread per column took 398 us for calc_r on 342 blocks of 32^3: 14 FP64
// operations a cell, and one block of 1024 threads per SM at a time.
template <int N, int VC, int MODE, int S>
struct ResStream {
  using R = PlaneRing<double, N, VC, S, true, (MODE == 0 ? 0 : 1)>;
  static constexpr int NT = 256;
  static constexpr size_t SMEM = R::SMEM;
  static constexpr int MINB = stream_minb<SMEM + 64, 4>();
};

template <int N, int VC, int MODE, int S>
__global__ void __launch_bounds__(256, (ResStream<N, VC, MODE, S>::MINB)) residual_stream_kernel(
    double* __restrict__ out, const double* __restrict__ x, const double* __restrict__ bb,
    const double* __restrict__ cf8, Geom g, int zc, double* __restrict__ partial, int* err) {
  using R = typename ResStream<N, VC, MODE, S>::R;
  constexpr int NT = 256, CPT = N * N / NT, LX = R::LX, LXY = R::LXY;
  extern __shared__ __align__(128) unsigned char smraw[];
  const int b = blockIdx.x, tid = threadIdx.x;
  const int64_t base = (int64_t)b * g.bstride + (int64_t)blockIdx.y * zc * LXY;
  R ring(smraw, zc);
  const double* C[1] = {bb};
  if (tid == 0) ring.start(x, C, base);
  double c[7];
#pragma unroll
  for (int q = 0; q < 7; q++) c[q] = cf8[(int64_t)b * 8 + q];
  int o[CPT];
#pragma unroll
  for (int k = 0; k < CPT; k++) {
    const int e = tid + k * NT;
    o[k] = R::at(e % N, e / N);
  }
  double acc = 0.0, none = 0.0;
  // products of the six neighbours and the cell's own -> its result
  auto finish = [&](int m, int q, const double* p, double centre) {
    if (MODE == 0) {
      double a = xadd(p[0], p[1]);
#pragma unroll
      for (int k = 2; k < 6; k++) a = xadd(a, p[k]);
      out[base + (int64_t)(VC + m) * LXY + q] = xadd(a, centre);
    } else {
      double r = ring.cp(m + 1, 0)[q];
#pragma unroll
      for (int k = 0; k < 6; k++) r = xsub(r, p[k]);
      r = xsub(r, centre);
      if (MODE == 1) out[base + (int64_t)(VC + m) * LXY + q] = r;
      else acc = __fma_rn(r, r, acc);
    }
  };
  __syncthreads();  // the ring's barriers are initialised
  bool ok;
  if (one_coefficient(c[1], c[2], c[3], c[4], c[5], c[6])) {
    ScaledPlanes<N, VC, NT, R> sp;
    ok = plane_walk(ring, x, C, base, err, tid, [&](int m) {
      if (m == 0) sp.begin(ring, c[1], o, tid);
      sp.take(ring, c[1], o, m, tid);
      const double* pc = ring.xp(m + 1);
#pragma unroll
      for (int k = 0; k < CPT; k++) {
        const int q = o[k];
        const double p[6] = {pc[q - 1], pc[q + 1], pc[q - LX], pc[q + LX], sp.pm[k], sp.pu[k]};
        finish(m, q, p, xmul(c[0], sp.xc[k]));
      }
      sp.shift();
    });
  } else {
    ok = plane_walk(ring, x, C, base, err, tid, [&](int m) {
      const double *xm = ring.xp(m), *xc = ring.xp(m + 1), *xu = ring.xp(m + 2);
#pragma unroll
      for (int k = 0; k < CPT; k++) {
        const int q = o[k];
        const double p[6] = {xmul(c[1], xc[q - 1]),  xmul(c[2], xc[q + 1]), xmul(c[3], xc[q - LX]),
                             xmul(c[4], xc[q + LX]), xmul(c[5], xm[q]),     xmul(c[6], xu[q])};
        finish(m, q, p, xmul(c[0], xc[q]));
      }
    });
  }
  if (MODE == 2) {
    // a copy that never arrived makes the sum NaN
    if (!ok) acc = __longlong_as_double(0x7ff8000000000000ll);
    kr_block_sums<1>(acc, none, reinterpret_cast<double*>(smraw + R::BAR_BYTES));
    if (tid == 0) partial[b * gridDim.y + blockIdx.y] = acc;
  }
}

template <int N, int VC, int MODE>
static cudaError_t residual_stream(double* out, const double* x, const double* b,
                                   const double* cf8, const Geom& g, double* partial, int* err,
                                   cudaStream_t st) {
  constexpr int S = N == 32 ? 4 : 6;
  using RS = ResStream<N, VC, MODE, S>;
  auto kern = residual_stream_kernel<N, VC, MODE, S>;
  static SharedMemory shared;
  if (cudaError_t e = shared.allow(kern, RS::SMEM)) return e;
  const int parts = kr_parts(g);
  kern<<<dim3(g.nb, parts), RS::NT, RS::SMEM, st>>>(out, x, b, cf8, g, N / parts, partial, err);
  return cudaGetLastError();
}

template <int MODE>
static cudaError_t residual_stream_mode(double* out, const double* x, const double* b,
                                        const double* cf8, const Geom& g, double* partial,
                                        int* err, cudaStream_t st) {
  if (g.nx == 32)
    return g.vc == 1 ? residual_stream<32, 1, MODE>(out, x, b, cf8, g, partial, err, st)
                     : residual_stream<32, 2, MODE>(out, x, b, cf8, g, partial, err, st);
  return g.vc == 1 ? residual_stream<16, 1, MODE>(out, x, b, cf8, g, partial, err, st)
                   : residual_stream<16, 2, MODE>(out, x, b, cf8, g, partial, err, st);
}

template <typename T>
cudaError_t launch_residual(T* out, const T* x, const T* b, Op<T> op, const Geom& g, int mode,
                            bool streamed, double* partial, int* err, cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  if constexpr (sizeof(T) == 8) {
    if (streamed) {
      if (mode == 0) return residual_stream_mode<0>(out, x, b, op.cf8, g, partial, err, st);
      if (mode == 1) return residual_stream_mode<1>(out, x, b, op.cf8, g, partial, err, st);
      return residual_stream_mode<2>(out, x, b, op.cf8, g, partial, err, st);
    }
  }
  if (cubic_fast(op, g)) {
    if (mode == 0) residual_cubic<T, 0>(out, x, b, op, g, partial, st);
    else if (mode == 1) residual_cubic<T, 1>(out, x, b, op, g, partial, st);
    else residual_cubic<T, 2>(out, x, b, op, g, partial, st);
    return cudaGetLastError();
  }
  if (mode == 0) return launch_sweep<T, 0>(out, x, b, op, g, T(0), partial, st);
  if (mode == 1) return launch_sweep<T, 1>(out, x, b, op, g, T(0), partial, st);
  return launch_sweep<T, 2>(out, x, b, op, g, T(0), partial, st);
}

// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) dot_partial_kernel(const T* __restrict__ x,
                                                          const T* __restrict__ y, Geom g,
                                                          double* __restrict__ partial) {
  constexpr int U = 8;
  __shared__ double red[256];
  const int b = blockIdx.x;
  const int64_t base = (int64_t)b * g.bstride;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  double acc = 0.0;
  for (int ij = threadIdx.x; ij < nx * ny; ij += blockDim.x) {
    const int i = ij % nx, j = ij / nx;
    int64_t p = base + g.at(i, j, 0);
    if constexpr (sizeof(T) == 4) {
      // float: the column's products summed in float-float where they are
      // exact there (2^-100 <= |x y| < 2^100: the product's error term is a
      // normal float), in double otherwise; GB300's FP64 rate would bound a
      // per-element FP64 accumulation.
      float s = 0.f, c = 0.f;
      double wide = 0.0;
      auto add = [&](float xv, float yv) {
        const ff q = two_prod(xv, yv);
        const float m = fabsf(q.hi);
        if (m >= 0x1p-100f && m < 0x1p100f) {
          const ff t = two_sum(s, q.hi);
          s = t.hi;
          c = __fadd_rn(c, __fadd_rn(t.lo, q.lo));
        } else if (xv != 0.f && yv != 0.f) {
          wide += (double)xv * (double)yv;
        }
      };
      // the loads of U planes before the first product (whose branch would
      // keep the next load behind it)
      int k = 0;
      for (; k + U <= nz; k += U, p += (int64_t)U * g.sz) {
        float xv[U], yv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          xv[u] = x[p + (int64_t)u * g.sz];
          yv[u] = y[p + (int64_t)u * g.sz];
        }
#pragma unroll
        for (int u = 0; u < U; u++) add(xv[u], yv[u]);
      }
      for (; k < nz; k++, p += g.sz) add(x[p], y[p]);
      acc += (double)s + (double)c + wide;
    } else {
      int k = 0;
      for (; k + U <= nz; k += U, p += (int64_t)U * g.sz) {
        T xv[U], yv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          xv[u] = x[p + (int64_t)u * g.sz];
          yv[u] = y[p + (int64_t)u * g.sz];
        }
#pragma unroll
        for (int u = 0; u < U; u++) acc += (double)xv[u] * (double)yv[u];
      }
      for (; k < nz; k++, p += g.sz) acc += (double)x[p] * (double)y[p];
    }
  }
  double none = 0.0;
  kr_block_sums<1>(acc, none, red);
  if (threadIdx.x == 0) partial[b] = acc;
}

template <typename T>
cudaError_t launch_dot_partial(const T* x, const T* y, const Geom& g, double* partial,
                               cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  // whole warps: kr_block_sums
  const int nt = (min(256, g.nx * g.ny) + 31) / 32 * 32;
  dot_partial_kernel<T><<<g.nb, nt, 0, st>>>(x, y, g, partial);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(1024) reduce_final_kernel(const double* __restrict__ partial,
                                                            int n, double* __restrict__ out) {
  __shared__ double red[32];
  constexpr int U = 8;  // loads of eight rounds before the first addition
  const int bd = blockDim.x;
  double acc = 0.0;
  int i = threadIdx.x;
  for (; i + (U - 1) * bd < n; i += U * bd) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = partial[i + u * bd];
#pragma unroll
    for (int u = 0; u < U; u++) acc += v[u];
  }
  for (; i < n; i += bd) acc += partial[i];
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) out[0] = acc;
}

cudaError_t launch_reduce_final(const double* partial, int n, double* out, cudaStream_t st) {
  reduce_final_kernel<<<1, 1024, 0, st>>>(partial, n, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CTA (b, z): planes [z zc, (z + 1) zc) of block b (sweep_chunk), the loads of
// U planes before the first store (z may be x or y: a cell reads only itself).
template <typename T, int KIND>
__global__ void __launch_bounds__(256) blas1_kernel(T* z, const T* x, const T* y, T a, T bc,
                                                    Geom g, int zc) {
  constexpr int U = 4;
  const int64_t base = (int64_t)blockIdx.x * g.bstride;
  const int nx = g.nx, ncol = g.nx * g.ny;
  const int z0 = blockIdx.y * zc, z1 = min(g.nz, z0 + zc);
  for (int ij = threadIdx.x; ij < ncol; ij += blockDim.x) {
    int64_t p = base + g.at(ij % nx, ij / nx, z0);
    auto planes = [&](auto vt) {
      constexpr int V = decltype(vt)::value;
      T zv[V], xv[V], yv[V];
#pragma unroll
      for (int u = 0; u < V; u++) {
        const int64_t q = p + (int64_t)u * g.sz;
        if (KIND != 2) zv[u] = z[q];
        if (KIND != 4) xv[u] = x[q];
        if (KIND == 2 || KIND == 3) yv[u] = y[q];
      }
#pragma unroll
      for (int u = 0; u < V; u++) {
        const int64_t q = p + (int64_t)u * g.sz;
        if (KIND == 0) z[q] = xadd(zv[u], xmul(a, xv[u]));                                // axpy
        else if (KIND == 1) z[q] = xadd(xv[u], xmul(a, zv[u]));                           // xpay
        else if (KIND == 2) z[q] = xadd(xmul(a, xv[u]), yv[u]);                           // axpyz
        else if (KIND == 3) z[q] = xadd(xadd(xmul(a, xv[u]), xmul(bc, yv[u])), zv[u]);    // axpbypz
        else z[q] = xmul(a, zv[u]);                                                      // scal
      }
      p += (int64_t)V * g.sz;
    };
    int k = z0;
    for (; k + U <= z1; k += U) planes(std::integral_constant<int, U>{});
    for (; k < z1; k++) planes(std::integral_constant<int, 1>{});
  }
}

template <typename T>
cudaError_t launch_blas1(int kind, T* z, const T* x, const T* y, T a, T b, const Geom& g,
                         cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  const int zc = sweep_chunk(g), th = column_threads(g);
  const dim3 grid(g.nb, (g.nz + zc - 1) / zc);
  switch (kind) {
    case 0: blas1_kernel<T, 0><<<grid, th, 0, st>>>(z, x, y, a, b, g, zc); break;
    case 1: blas1_kernel<T, 1><<<grid, th, 0, st>>>(z, x, y, a, b, g, zc); break;
    case 2: blas1_kernel<T, 2><<<grid, th, 0, st>>>(z, x, y, a, b, g, zc); break;
    case 3: blas1_kernel<T, 3><<<grid, th, 0, st>>>(z, x, y, a, b, g, zc); break;
    default: blas1_kernel<T, 4><<<grid, th, 0, st>>>(z, x, y, a, b, g, zc); break;
  }
  return cudaGetLastError();
}

// The ghost planes in z (and the ghost rows in y) of a brick: contiguous but for
// the interior rows, one warp per piece.
template <typename T>
__global__ void __launch_bounds__(256) copy_frame_kernel(T* __restrict__ dst,
                                                         const T* __restrict__ src, Geom g,
                                                         int rows) {
  const int64_t base = (int64_t)blockIdx.x * g.bstride;
  T* d = dst + base;
  const T* s = src + base;
  const int ends = g.vc * g.sz;                // the ghost planes at either end
  const int hi = (g.vc + g.nz) * g.sz;
  for (int e = threadIdx.x; e < ends; e += blockDim.x) {
    d[e] = s[e];
    d[hi + e] = s[hi + e];
  }
  if (!rows) return;
  const int n = g.vc * g.sy, up = (g.vc + g.ny) * g.sy;
  for (int z = g.vc + (threadIdx.x >> 5); z < g.vc + g.nz; z += blockDim.x >> 5)
    for (int e = threadIdx.x & 31; e < n; e += 32) {
      d[z * g.sz + e] = s[z * g.sz + e];
      d[z * g.sz + up + e] = s[z * g.sz + up + e];
    }
}

template <typename T>
cudaError_t launch_copy_frame(T* dst, const T* src, const Geom& g, bool rows, cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  copy_frame_kernel<T><<<g.nb, 256, 0, st>>>(dst, src, g, rows ? 1 : 0);
  return cudaGetLastError();
}

template <typename T>
__global__ void fill_kernel(T* __restrict__ x, int64_t n, T v) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    x[e] = v;
}

template <typename T>
cudaError_t launch_fill(T* x, int64_t n, T v, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  fill_kernel<T><<<(int)blocks, 256, 0, st>>>(x, n, v);
  return cudaGetLastError();
}

// Seeded uniform values in [lo, hi) on the interior of blocks [b0, b0+nb)
// (ghosts untouched): value of interior cell c of local block l is a
// splitmix64 hash of (seed, l, c) scaled to the interval, so a block set
// gets the same values wherever it sits in a larger mesh.
__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

template <typename T>
__global__ void __launch_bounds__(256) fill_random_kernel(T* __restrict__ x, Geom g, int b0,
                                                          int nb, uint64_t seed, double lo,
                                                          double hi) {
  const int64_t cells = (int64_t)g.nx * g.ny * g.nz;
  const int64_t total = cells * nb;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t l = e / cells, c = e - l * cells;
    const int i = (int)(c % g.nx), j = (int)((c / g.nx) % g.ny), k = (int)(c / ((int64_t)g.nx * g.ny));
    const uint64_t h = splitmix64(seed * 0x100000001b3ull ^ splitmix64((uint64_t)l * (uint64_t)cells + (uint64_t)c));
    const double u = (double)(h >> 11) * 0x1p-53;  // [0, 1)
    x[(int64_t)(b0 + l) * g.bstride + g.at(i, j, k)] = (T)(lo + (hi - lo) * u);
  }
}

template <typename T>
cudaError_t launch_fill_random(T* x, const Geom& g, int b0, int nb, uint64_t seed, double lo,
                               double hi, cudaStream_t st) {
  const int64_t total = (int64_t)g.nx * g.ny * g.nz * nb;
  if (total == 0) return cudaSuccess;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  fill_random_kernel<T><<<(int)blocks, 256, 0, st>>>(x, g, b0, nb, seed, lo, hi);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Boundary folding (SolverTest bca.f90:12-394, applied per block by
// BlockScalar3D::ImposeBoundaryCondition, BlockScalar3D.h:208-215).  For an
// outer face with neighbour coefficient A_nb and value xc:
//   Dirichlet  Ap -= A_nb;  b = (T)((double)b - (double)(A_nb*xc) * 2);  A_nb = 0
//   Neumann    Ap += A_nb;  b += A_nb*xc (minus faces) or -= (plus faces);  A_nb = 0
// with A_nb*xc rounded to T first (Fortran `real` operands, then the
// double-precision 2.0d0 factor).  One launch per axis; each thread takes one
// cell of the face plane and folds its minus face before its plus face.
template <typename T>
__device__ __forceinline__ void fold_cell(T* __restrict__ Ap, T* __restrict__ An,
                                          T* __restrict__ b, int q, int code, T xc, bool minus) {
  const T a = An[q];
  const T p = xmul(a, xc);
  if (code == 1) {
    Ap[q] = xsub(Ap[q], a);
    b[q] = to_t<T>(xsub((double)b[q], xmul((double)p, 2.0)));
  } else {
    Ap[q] = xadd(Ap[q], a);
    b[q] = minus ? xadd(b[q], p) : xsub(b[q], p);
  }
  An[q] = (T)0;
}

template <typename T>
__global__ void __launch_bounds__(256) fold_axis_kernel(FoldPtrs<T> p, Geom g, int ax,
                                                         const int* __restrict__ code,
                                                         const double* __restrict__ xcv) {
  const int blk = blockIdx.x;
  const int fm = 2 * ax, fp = 2 * ax + 1;
  const int cm = code[blk * 6 + fm], cp = code[blk * 6 + fp];
  if (cm == 0 && cp == 0) return;
  const T xm = (T)xcv[blk * 6 + fm], xp = (T)xcv[blk * 6 + fp];
  const int n[3] = {g.nx, g.ny, g.nz};
  const int u = ax == 0 ? 1 : 0, v = ax == 2 ? 1 : 2;  // the plane's axes
  const int64_t base = (int64_t)blk * g.bstride;
  T* Ap = p.A[0] + base;
  T* Am = p.A[1 + 2 * ax] + base;
  T* Aq = p.A[2 + 2 * ax] + base;
  T* b = p.b + base;
  for (int e = threadIdx.x; e < n[u] * n[v]; e += blockDim.x) {
    int c[3];
    c[u] = e % n[u];
    c[v] = e / n[u];
    if (cm) {
      c[ax] = 0;
      fold_cell(Ap, Am, b, g.at(c[0], c[1], c[2]), cm, xm, true);
    }
    if (cp) {
      c[ax] = n[ax] - 1;
      fold_cell(Ap, Aq, b, g.at(c[0], c[1], c[2]), cp, xp, false);
    }
  }
}

template <typename T>
cudaError_t launch_fold_boundary(FoldPtrs<T> p, const Geom& g, const int* code, const double* xc,
                                 cudaStream_t st) {
  if (g.nb == 0) return cudaSuccess;
  for (int ax = 0; ax < 3; ax++) {
    fold_axis_kernel<T><<<g.nb, 256, 0, st>>>(p, g, ax, code, xc);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Mixed precision helpers: interior FP64 -> FP32 (residual hand-off) and
// x64 += (double) d32 (correction accumulation).  Both fields share vc.
__global__ void __launch_bounds__(256) convert_kernel(float* __restrict__ dst,
                                                      const double* __restrict__ src, Geom g64,
                                                      Geom g32) {
  const int b = blockIdx.x;
  const int nx = g64.nx, ny = g64.ny, nz = g64.nz;
  for (int ij = threadIdx.x; ij < nx * ny; ij += blockDim.x) {
    const int i = ij % nx, j = ij / nx;
    for (int k = 0; k < nz; k++) {
      const int q = g64.at(i, j, k);
      dst[(int64_t)b * g32.bstride + q] = __double2float_rn(src[(int64_t)b * g64.bstride + q]);
    }
  }
}

__global__ void __launch_bounds__(256) accumulate_kernel(double* __restrict__ x,
                                                         const float* __restrict__ d, Geom g64,
                                                         Geom g32) {
  const int b = blockIdx.x;
  const int nx = g64.nx, ny = g64.ny, nz = g64.nz;
  for (int ij = threadIdx.x; ij < nx * ny; ij += blockDim.x) {
    const int i = ij % nx, j = ij / nx;
    for (int k = 0; k < nz; k++) {
      const int q = g64.at(i, j, k);
      const int64_t p = (int64_t)b * g64.bstride + q;
      x[p] = x[p] + (double)d[(int64_t)b * g32.bstride + q];
    }
  }
}

cudaError_t launch_convert_f64_to_f32(float* dst, const double* src, const Geom& g64,
                                      const Geom& g32, cudaStream_t st) {
  if (g64.nb == 0) return cudaSuccess;
  convert_kernel<<<g64.nb, min(256, g64.nx * g64.ny), 0, st>>>(dst, src, g64, g32);
  return cudaGetLastError();
}

cudaError_t launch_accumulate_f32_into_f64(double* x, const float* d, const Geom& g64,
                                           const Geom& g32, cudaStream_t st) {
  if (g64.nb == 0) return cudaSuccess;
  accumulate_kernel<<<g64.nb, min(256, g64.nx * g64.ny), 0, st>>>(x, d, g64, g32);
  return cudaGetLastError();
}

#define INST(T)                                                                              \
  template cudaError_t launch_copy_frame<T>(T*, const T*, const Geom&, bool, cudaStream_t); \
  template cudaError_t launch_jacobi<T>(T*, const T*, const T*, Op<T>, const Geom&, T,      \
                                        cudaStream_t);                                      \
  template cudaError_t launch_residual<T>(T*, const T*, const T*, Op<T>, const Geom&, int, bool, \
                                          double*, int*, cudaStream_t);                           \
  template cudaError_t launch_dot_partial<T>(const T*, const T*, const Geom&, double*,      \
                                             cudaStream_t);                                 \
  template cudaError_t launch_blas1<T>(int, T*, const T*, const T*, T, T, const Geom&,      \
                                       cudaStream_t);                                       \
  template cudaError_t launch_fill<T>(T*, int64_t, T, cudaStream_t);                       \
  template cudaError_t launch_fill_random<T>(T*, const Geom&, int, int, uint64_t, double,  \
                                             double, cudaStream_t);                         \
  template cudaError_t launch_fold_boundary<T>(FoldPtrs<T>, const Geom&, const int*,        \
                                               const double*, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace bcmg

// ---------------------------------------------------------------------------
// Inner product without any allocation, for callers that cannot call
// cudaMalloc: host code embedded in a larger application or framework that
// owns every device allocation (its own pool or allocator, nothing else may
// allocate beside it), which would otherwise have to hand this library a
// scratch buffer it does not know how to size.  The per-block partial sums,
// which bcmg_dot keeps in a per-context buffer, live here in one file-scope
// device array of fixed capacity that every GPU loading this library holds
// until the process exits.
#include <cuda.h>

#include <mutex>

#include "bcmg.h"

namespace {

__device__ __align__(256) double g_noalloc_partials[BCMG_NOALLOC_MAX_BLOCKS];

// Device address of g_noalloc_partials, looked up with cudaGetSymbolAddress
// once per device and CUDA context (with that device current).  In host code
// the array's name is only a host-side stand-in, never a device address.
// The context id (cuCtxGetId, unique for the life of the process) keys the
// cache, so that after a cudaDeviceReset or a re-created primary context the
// address is looked up again instead of reusing one that is no longer mapped.
constexpr int kMaxDevices = 64;
struct PartialsAddr {
  unsigned long long ctx_id;
  double* ptr;
};
PartialsAddr g_partials_addr[kMaxDevices] = {};
std::mutex g_partials_mu;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// Driver entry points through the runtime (the library links only cudart).
bool current_context_id(unsigned long long* id) {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  if (!get_current || !get_id) {
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) !=
            cudaSuccess || q1 != cudaDriverEntryPointSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) !=
            cudaSuccess || q2 != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return false;
    }
    get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
    get_id = reinterpret_cast<CtxGetIdFn>(f2);
  }
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
  return get_id(ctx, id) == CUDA_SUCCESS;
}

}  // namespace

extern "C" BCMG_API int bcmg_dot_noalloc(int dtype, const void* x, const void* y, int nb, int nx,
                                         int ny, int nz, int vc, int64_t block_stride,
                                         double* result, void* stream) {
  using namespace bcmg;
  if ((dtype != BCMG_F32 && dtype != BCMG_F64) || !x || !y || !result) return BCMG_USAGE;
  if (nb < 0 || nx < 1 || ny < 1 || nz < 1 || vc < 1) return BCMG_USAGE;
  // every brick index the kernels form is an int: the padded plane and the
  // padded brick must fit in int32
  const int64_t sy = (int64_t)nx + 2 * (int64_t)vc;
  const int64_t plane = sy * ((int64_t)ny + 2 * (int64_t)vc);
  const int64_t brick = plane * ((int64_t)nz + 2 * (int64_t)vc);
  if (sy > INT32_MAX || plane > INT32_MAX || brick > INT32_MAX) return BCMG_USAGE;
  if (block_stride < brick) return BCMG_USAGE;
  if (nb > BCMG_NOALLOC_MAX_BLOCKS) return BCMG_SCRATCH_LIMIT;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return BCMG_NO_DEVICE;
  }
  if (dev < 0 || dev >= kMaxDevices) return BCMG_USAGE;
  double* part;
  {
    std::lock_guard<std::mutex> lock(g_partials_mu);
    unsigned long long ctx_id = 0;
    const bool have_ctx = current_context_id(&ctx_id);
    if (!have_ctx || !g_partials_addr[dev].ptr || g_partials_addr[dev].ctx_id != ctx_id) {
      // set-up for this device and context (the lookup also makes the
      // device's primary context current on a thread that has none yet)
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_partials) != cudaSuccess || !p) {
        cudaGetLastError();
        return BCMG_CUDA_ERROR;
      }
      if (!current_context_id(&ctx_id)) return BCMG_CUDA_ERROR;
      g_partials_addr[dev].ptr = static_cast<double*>(p);
      g_partials_addr[dev].ctx_id = ctx_id;
    }
    part = g_partials_addr[dev].ptr;
  }
  if (nb == 0) {
    // an empty mesh: the reduction of zero partials writes 0
    return launch_reduce_final(part, 0, result, (cudaStream_t)stream) == cudaSuccess
               ? BCMG_SUCCESS : BCMG_CUDA_ERROR;
  }
  Geom g;
  g.nx = nx; g.ny = ny; g.nz = nz; g.vc = vc;
  g.sy = (int)sy;
  g.sz = (int)plane;
  g.off0 = (int)((1 + sy + plane) * vc);
  g.bstride = block_stride;
  g.nb = nb;
  cudaError_t e = dtype == BCMG_F64
      ? launch_dot_partial<double>((const double*)x, (const double*)y, g, part, (cudaStream_t)stream)
      : launch_dot_partial<float>((const float*)x, (const float*)y, g, part, (cudaStream_t)stream);
  if (e == cudaSuccess) e = launch_reduce_final(part, nb, result, (cudaStream_t)stream);
  return e == cudaSuccess ? BCMG_SUCCESS : BCMG_CUDA_ERROR;
}
