// sor_stream.cuh -- fused red-black SOR pass of blocks too large to stage whole,
// or of no special shape: one CTA per block streams the brick's z-planes (and
// the source's) through a ring in shared memory and writes the pass's result
// once, then the ghost values it feeds (push form).
//
// Both colours in one walk: colour 0 of plane t reads colour-1 cells of planes
// t-1, t, t+1 as they were, colour 1 of plane t-2 reads colour-0 cells of planes
// t-3, t-2, t-1 as updated; neither touches what the other reads, so phase t
// does both with one CTA barrier before it.  (sor1/Solver.cpp:132-153,
// sor2/Solver.cpp:136-160: ghosts are read as they were before the pass.)
//
// Unit u of the ring is plane u - 1 of the block, rows [-1, ny] (and, for interior
// planes, the source's rows [0, ny)), one bulk copy each, widened to
// 16-byte bounds: a brick plane is a multiple of 16 bytes for every even block
// shape.  Unit t-3 is last read in phase t-1; its slot then takes unit t-3+S.
// Waits are bounded as in stream.cuh.
//
// A block may be split over a cluster of 2, 4 or 8 CTAs (fewer than two
// blocks per SM leave it half idle, sor_split): each makes colour 1 of its
// planes [k0, k1) and colour 0 of those and one more on either side -- the colour
// its neighbour makes of the same values of A -- writes its planes, and after a
// cluster barrier its share of the ghosts.
//
// Bound: HBM in FP32, the FP64 pipe in FP64.  The brick staged whole left one
// CTA of 256 threads per SM for 32^3 (170 us an iteration on 18.8 M cells, FP32)
// and the general kernel walked cells with a division each (124 us on 7.9 M
// cells of 24^3 blocks).
#pragma once
#include "attr.h"
#include "bulk.cuh"
#include "cells.cuh"
#include "tile.cuh"

namespace bcmg {

// N > 0: cubic blocks of edge N and ghost width VC (compile-time offsets, the
// specialised pushes); N = 0: any shape.
template <typename T, int FORM, int N, int VC>
__global__ void __launch_bounds__(256, (sizeof(T) == 4 ? 4 : 2))
    sor_stream_kernel(const T* __restrict__ A, T* Bf, const T* __restrict__ S, Geom g, SorArgs a,
                      SorRing r) {
  extern __shared__ __align__(128) unsigned char smraw[];
  const int rank = blockIdx.x % r.ranks, b = blockIdx.x / r.ranks;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int nx = N ? N : g.nx, ny = N ? N : g.ny, nz = N ? N : g.nz, vc = N ? VC : g.vc;
  const int sy = N ? N + 2 * VC : g.sy, sz = N ? (N + 2 * VC) * (N + 2 * VC) : g.sz;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smraw);
  unsigned char* ring = smraw + 128;
  const int64_t base = (int64_t)b * g.bstride;
  const unsigned char* Ab = reinterpret_cast<const unsigned char*>(A + base);
  const unsigned char* Sb = FORM == 2 ? reinterpret_cast<const unsigned char*>(S + base) : nullptr;
  T* fb = Bf + base;
  // this CTA's planes, and the planes [c0, c0 + n0) of which it makes colour 0;
  // unit u is plane c0 - 1 + u
  const int zc = (nz + r.ranks - 1) / r.ranks, k0 = rank * zc, k1 = min(nz, k0 + zc);
  const int c0 = max(0, k0 - 1), n0 = min(nz, k1 + 1) - c0;
  const int nu = n0 + 2;
  auto issue = [&](int u, int s) {
    const bool cells = FORM == 2 && u >= 1 && u <= n0;
    unsigned char* d = ring + (size_t)s * r.slot;
    const size_t plane = (size_t)(vc - 1 + c0 + u) * sz * sizeof(T);
    mbar_expect_tx(&bar[s], r.xbytes + (cells ? r.sbytes : 0));
    bulk_g2s(d, Ab + plane + r.xlo, r.xbytes, &bar[s]);
    if (cells) bulk_g2s(d + r.xbytes, Sb + plane + r.slo, r.sbytes, &bar[s]);
  };
  int issued = min(r.slots, nu);
  if (tid == 0) {
    for (int s = 0; s < r.slots; s++) mbar_init(&bar[s], 1);
    mbar_fence_init();
    for (int u = 0; u < issued; u++) issue(u, u);
  }
  // block constants while the copies run
  SorCell<T, FORM> cell;
  cell.init(a, b);
  const unsigned dmask = dirichlet_mask(a, b);
  const int p0 = a.push.ptr[b], p1 = a.push.ptr[b + 1];
  // this thread's cell pairs (x = 2 i2, 2 i2 + 1) of a plane: tid, tid + nt, ...
  const int hx = nx / 2, np = hx * ny;
  const int j0 = tid / hx, i0 = tid - j0 * hx;
  const int dj = nt / hx, di = nt - dj * hx;
  const int ox = vc + vc * sy - r.xlo / (int)sizeof(T);  // x plane's index of (0, 0)
  const int os = vc + vc * sy - r.slo / (int)sizeof(T);
  auto xplane = [&](int s) { return reinterpret_cast<T*>(ring + (size_t)s * r.slot) + ox; };
  auto splane = [&](int s) {
    return reinterpret_cast<const T*>(ring + (size_t)s * r.slot + r.xbytes) + os;
  };
  bool ok = true;
  auto walk = [&](auto&& upd) {
    // ring slots of units t-2 .. t+2
    int s_2 = 0, s_1 = 0, s0 = 0, s1 = 1, s2 = 2;
    unsigned ph = 0;  // phase parity of unit t+2
    for (int t = 0; t < n0 + 2; t++) {
      if (tid == 0 && t < n0) {
        if (t == 0) ok = mbar_wait_quiet(&bar[0], 0, a.err) && mbar_wait_quiet(&bar[1], 0, a.err);
        ok = ok && mbar_wait_quiet(&bar[s2], ph, a.err);
      }
      if (!__syncthreads_and(ok)) {
        ok = false;
        break;
      }
      // the slot of unit t-3 is free
      if (tid == 0 && t >= 3 && t - 3 + r.slots < nu) {
        int s = s_2 - 1;
        if (s < 0) s += r.slots;
        issue(t - 3 + r.slots, s);
        issued = t - 2 + r.slots;
      }
      if (t < n0) {  // colour 0 of plane c0 + t
        const T* xm = xplane(s0);
        T* xc = xplane(s1);
        const T* xu = xplane(s2);
        const T* sp = splane(s1);
        for (int e = tid, j = j0, i2 = i0; e < np; e += nt) {
          const int q = j * sy + 2 * i2 + ((j + c0 + t) & 1);
          const T sw = xadd(xc[q - 1], xc[q + 1]);
          const T ss = xadd(xc[q - sy], xc[q + sy]);
          const T sb = xadd(xm[q], xu[q]);
          xc[q] = upd(xc[q], sw, ss, sb, FORM == 2 ? sp[q] : T(0));
          i2 += di;
          j += dj;
          if (i2 >= hx) { i2 -= hx; j++; }
        }
      }
      const int k = c0 + t - 2;
      if (k >= k0 && k < k1) {  // colour 1 of plane k, and its rows to B
        const T* xm = xplane(s_2);
        const T* xc = xplane(s_1);
        const T* xu = xplane(s0);
        const T* sp = splane(s_1);
        T* out = fb + (int64_t)(vc + k) * sz + vc * sy + vc;
        for (int e = tid, j = j0, i2 = i0; e < np; e += nt) {
          const int par = (1 + j + k) & 1, q = j * sy + 2 * i2 + par;
          const T sw = xadd(xc[q - 1], xc[q + 1]);
          const T ss = xadd(xc[q - sy], xc[q + sy]);
          const T sb = xadd(xm[q], xu[q]);
          const T v = upd(xc[q], sw, ss, sb, FORM == 2 ? sp[q] : T(0));
          const int p = j * sy + 2 * i2;
          const T o = xc[p + (par ^ 1)];
          out[p] = par ? o : v;
          out[p + 1] = par ? v : o;
          i2 += di;
          j += dj;
          if (i2 >= hx) { i2 -= hx; j++; }
        }
      }
      fence_proxy_async_smem();  // colour 0's stores, before the slot is refilled
      s_2 = t >= 1 ? s_1 : 0;
      s_1 = s0;
      s0 = s1;
      s1 = s2;
      if (++s2 == r.slots) { s2 = 0; ph ^= 1; }
    }
  };
  __syncthreads();  // the barriers are initialised
  if constexpr (sizeof(T) == 8 && FORM == 2) {
    if (cell.power_of_two())
      walk([&](T f, T x, T y, T z, T s) { return cell.scaled(f, x, y, z, s); });
    else
      walk([&](T f, T x, T y, T z, T s) { return cell(f, x, y, z, s); });
  } else {
    walk([&](T f, T x, T y, T z, T s) { return cell(f, x, y, z, s); });
  }
  if (!ok) {
    // a copy never arrived (the error word says so): wait, bounded, for the
    // last unit issued into each slot
    if (tid == 0)
      for (int s = 0; s < r.slots; s++) {
        const int u = issued - 1 - ((issued - 1 - s) % r.slots + r.slots) % r.slots;
        if (u >= 0) mbar_wait_quiet(&bar[s], (unsigned)(u / r.slots) & 1u, nullptr);
      }
    __syncthreads();
  }
  // the block's new interior is in its brick, seen by the CTA, or the cluster
  if (r.ranks > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
  else
    __syncthreads();
  if (!ok) return;
  // Dirichlet ghosts: g = 2v - f, and the second layer of the bcx form
  if (dmask) {
    const double* dval = a.bc.value + b * 6;
    for (int fc = 0; fc < 6; fc++) {
      if (!((dmask >> fc) & 1)) continue;
      const int ax = fc >> 1, minus = (fc & 1) == 0;
      const int d0 = ax == 0 ? ny : nx, d1 = ax == 2 ? ny : nz, nn = ax == 0 ? nx : ax == 1 ? ny : nz;
      double v = dval[fc];
      if (a.bc.bcx) v = (double)(T)v;
      const double v2 = xmul(2.0, v);
      const int st0 = ax == 0 ? sy : 1, st1 = ax == 2 ? sy : sz, stn = ax == 0 ? 1 : ax == 1 ? sy : sz;
      const int in = minus ? 0 : nn - 1, gh = minus ? -1 : nn, g2 = minus ? -2 : nn + 1;
      const int o = vc * (1 + sy + sz);
      for (int e = tid + rank * nt; e < d0 * d1; e += nt * r.ranks) {
        int q1, q0;
        divmod(e, d0, q1, q0);
        const int at = o + q0 * st0 + q1 * st1;
        fb[at + gh * stn] = to_t<T>(xsub(v2, (double)fb[at + in * stn]));
        if (a.bc.bcx && vc >= 2) fb[at + g2 * stn] = (T)v;
      }
    }
  }
  if constexpr (N > 0) {
    for (int q = p0 + ((tid + rank * nt) >> 5); q < p1; q += (nt >> 5) * r.ranks) {
      const VcTask t = a.push.tasks[q];
      push_dispatch<T, N, VC, BrickTile<T, N, VC>, 4>(t, Bf + (int64_t)t.dst * g.bstride, g, fb,
                                                      tid & 31);
    }
  } else {
    const Acc<T> src{fb, g.sy, g.sz, g.off0};
    const int es = entry_shift(g);
    for (int q = p0 + ((tid + rank * nt) >> es); q < p1; q += (nt >> es) * r.ranks) {
      const VcTask t = a.push.tasks[q];
      task_apply<T>(t, Bf + (int64_t)t.dst * g.bstride, g, src, 0.0, tid & ((1 << es) - 1),
                    1 << es);
    }
  }
}

// Whether the streamed pass covers a launch: one inner pass, a ring within
// shared memory, 16-byte aligned bricks.
template <typename T>
static bool sor_stream_ok(const Geom& g, const T* A, const T* s, int n_inner) {
  return sor_streams(g, s != nullptr, n_inner, sizeof(T)) &&
         ((size_t)g.bstride * sizeof(T)) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(s) % 16 == 0;
}

// CTAs per block: two, four or eight until there are three per SM in FP64 and for
// 128-thread planes, two in FP32, each with a share of six planes or more (the last
// one's may be smaller; a CTA makes colour 0 of two planes more than its own).  342
// blocks split in two: FP64 24^3 287 -> 233 us an iteration, 32^3 443 -> 394, FP32
// 8x6x24 36 -> 26 but 28^3 78 -> 85; 575 blocks: FP64 24^3 302 -> 334, FP32 69 -> 83.
// FP64 with 256 threads has two CTAs on an SM at a time: blocks, or halves of them,
// that come close to two per SM are left at that (24^3, us an iteration by CTAs per
// block 1 / 2 / 4: 152 blocks 84, 70, 97; 216 115, 127, 120; 304 118, 132, 167; 32^3:
// 152 blocks 130, 123, 157; 304 225, 235, 277).
inline int sor_split(const Geom& g, const SorRing& ring, size_t es) {
  if (es == 8 && ring.threads == 256) {
    if (g.nb <= 304 && g.nb >= 228) return 1;
    if (2 * g.nb <= 304 && 2 * g.nb >= 190 && g.nz >= 12) return 2;
  }
  const int want = (es == 8 || ring.threads == 128 ? 3 : 2) * 152;
  int r = 1;
  while (r < 8 && g.nb * r < want && g.nz >= 2 * r * 6) r *= 2;
  return r;
}

template <typename T, int FORM, int N, int VC>
static cudaError_t sor_stream_one(const T* A, T* B, const T* s, const Geom& g, const SorArgs& a,
                                  cudaStream_t st) {
  auto kern = sor_stream_kernel<T, FORM, N, VC>;
  static SharedMemory shared;
  if (cudaError_t e = shared.allow(kern, kSorMaxSmem)) return e;
  SorRing r = SorRing::make(g, FORM == 2, sizeof(T));
  r.ranks = sor_split(g, r, sizeof(T));
  return launch_dependent(kern, g.nb * r.ranks, r.threads, r.bytes(), st, false, r.ranks, A, B, s,
                          g, a, r);
}

template <typename T, int FORM>
static cudaError_t launch_sor_stream(const T* A, T* B, const T* s, const Geom& g,
                                     const SorArgs& a, cudaStream_t st) {
  if (g.nx == 32 && g.ny == 32 && g.nz == 32 && g.vc == 1)
    return sor_stream_one<T, FORM, 32, 1>(A, B, s, g, a, st);
  if (g.nx == 32 && g.ny == 32 && g.nz == 32 && g.vc == 2)
    return sor_stream_one<T, FORM, 32, 2>(A, B, s, g, a, st);
  return sor_stream_one<T, FORM, 0, 0>(A, B, s, g, a, st);
}

}  // namespace bcmg
