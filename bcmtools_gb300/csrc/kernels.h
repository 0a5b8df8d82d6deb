// kernels.h -- internal launcher declarations shared by the C ABI and the
// kernel translation units.  Not part of the public interface.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "krylov.cuh"

namespace bcmg {

// log2 of the lanes that share one face-table entry in the kernels for any block
// shape: a warp, or for small blocks the power of two that holds the largest
// ghost box (vc cells by the largest face), so that a warp takes several
// entries.  With a warp each, 2^3 blocks left 28 of 32 lanes idle in every FP64
// instruction (8.0 us an iteration of 456 such blocks).
__host__ __device__ inline int entry_shift(const Geom& g) {
  const int xy = g.nx * g.ny, yz = g.ny * g.nz, xz = g.nx * g.nz;
  const int most = g.vc * (xy > yz ? (xy > xz ? xy : xz) : (yz > xz ? yz : xz));
  int l = 5;
  while (l > 0 && (1 << (l - 1)) >= most) l--;
  return l;
}

// Up to 12 contiguous slices of the face table (4 kinds x 3 axes) selected
// by one launch; prefix[q] is the first warp of slice q.
struct VcRanges {
  int start[12];
  int prefix[13];
  int n;
};

template <typename T>
cudaError_t launch_vc_gather(T* data, const Geom& g, const VcTable& tab, const VcRanges& rg,
                             cudaStream_t st);

// Block Dirichlet description for the SOR kernel.
struct BlockBc {
  const int* type;      // [nb*6] BCMG_BC_*
  const double* value;  // [nb*6]
  int bcx;              // second ghost layer = v when vc >= 2
  // [nb*8] 2v (v rounded to float first in the bcx form) as a float where
  // that is exact, else NaN: lets float sweeps form 2v - f in one float
  // subtraction (tile_dirichlet)
  const float* v2f;
};

// Incoming ghost source of one face of one block (the pull form): kind -1
// (no neighbour), VC_COPY / VC_C2F (src[0], sub = the neighbour's subface)
// or VC_F2C (src[s] the fine neighbour on subface s).
struct FaceIn {
  int src[4];
  int kind;
  int sub;
};

// Per-block descriptor of the pull-form sweeps.  csrc[f]: the same-level
// neighbour on face f; for a face fed by a coarser block (flag bit
// bi_c2f_bit(f)) coarse block * 4 + this block's subface on it (the reader
// interpolates those ghosts from the coarse interior); for a face fed by
// finer blocks its slot in the side buffer of first-layer F2C ghosts; or -1.
// flags: bit f the face is fed by a neighbour (BI_FED << f), bit 8+f by a
// same-level one (BI_COPY << f), bit 16+f it carries a Dirichlet condition,
// bits 24..30 the number of F2C entries this block feeds (listed from
// out_begin).
struct BlockInfo {
  int csrc[6];
  int flags;
  int out_begin;
};
enum : unsigned { BI_FED = 1u, BI_COPY = 1u << 8, BI_DIR_SHIFT = 16, BI_OUT_SHIFT = 24 };
constexpr int kMaxOutEntries = 24;  // 6 faces x 4 finer neighbours
// Flag bit of a face fed by a coarser block (bits 6-7, 14-15, 22-23 are free).
__host__ __device__ constexpr int bi_c2f_bit(int f) { return f < 2 ? 6 + f : f < 4 ? 12 + f : 18 + f; }

// Outgoing ghost entries of every block (face-table entries grouped by source
// block, CSR): the entries a fused sweep CTA writes from shared memory.
struct PushTable {
  const int* ptr;        // [nb+1]
  const VcTask* tasks;   // entries with src == block, destination's view
  const unsigned char* fed;  // [nb] bit f: some neighbour writes face f's ghosts
  const FaceIn* in;          // [nb*6] ghost sources of each face (pull form)
  const BlockInfo* info;     // [nb] descriptors of the pull form
  const VcTask* out_tasks;   // F2C entries by source block (pull form)
  const void* side_in;       // first-layer F2C ghosts of the input
  void* side_out;            // ... of the output, written by their sources
  // x-face layers of the pipelined pull form, 2*N*N per block: block b's
  // columns x = 0 and x = N-1 (cell (y, z) at z*N + y) as the input had them,
  // and as the output has them (written by the launch that writes b)
  const void* xf_in;
  void* xf_out;
};


// Fewest CTAs the streamed 32^3 kernels should have: below, a block's planes are
// split over a cluster of them.
constexpr int kSplitCtas = 152 * 4;
constexpr size_t kSorMaxSmem = 200 * 1024;
// Dynamic shared memory one CTA may use (227 KB on sm_100-class GPUs).
constexpr size_t kPipeMaxSmem = 227 * 1024;

// Ring of the streamed red-black SOR pass (sor_stream.cuh): one unit holds rows
// [-1, ny] of a plane and, with a source, the source's rows [0, ny), each
// widened to 16-byte bounds.
struct SorRing {
  int xlo, xbytes;  // first byte and bytes of the rows of a brick plane
  int slo, sbytes;
  int slot, slots;  // bytes of a unit, units in shared memory
  int threads;      // of the CTA
  int ranks;        // CTAs per block (a cluster)
  static SorRing make(const Geom& g, bool src, size_t es) {
    SorRing r;
    r.ranks = 1;
    const int row = g.sy * (int)es;
    r.xlo = (g.vc - 1) * row / 16 * 16;
    r.xbytes = ((g.vc + g.ny + 1) * row + 15) / 16 * 16 - r.xlo;
    r.slo = g.vc * row / 16 * 16;
    r.sbytes = src ? ((g.vc + g.ny) * row + 15) / 16 * 16 - r.slo : 0;
    r.slot = r.xbytes + r.sbytes;
    // Planes of at most 128 cell pairs take 128 threads and a ring of eight per
    // SM, larger ones 256 and four per SM; six slots at least (one in flight)
    r.threads = g.nx / 2 * g.ny <= 128 ? 128 : 256;
    const int fit = (r.threads == 128 ? 27 : 55) * 1024 / r.slot;
    r.slots = fit < 6 ? 6 : fit > 16 ? 16 : fit;
    if (r.slots > g.nz + 2 && g.nz + 2 >= 6) r.slots = g.nz + 2;
    return r;
  }
  size_t bytes() const { return 128 + (size_t)slots * slot; }
};
// Whether that pass covers a run: one inner pass, whole 16-byte planes, a ring
// within shared memory.  FP32 blocks of up to 64 cells stay staged whole up to four
// per SM (288 blocks of 4^3: 7.4 us an iteration, streamed 8.8; 1408: 19.0 and 14.5),
// FP64 blocks of up to 256 cells stay staged whole (575
// blocks of 4^3: 17.9 us an iteration, streamed 20.1), so do many with planes of
// less than 40 cell pairs (8x6x24, 2491 blocks: 181 and 197; 575: 64 and 62), and
// bricks too large for that are swept in place unless the rounds of 256 threads
// over a plane are nearly full (28^3: 410 us in place, 462 streamed at 77 %;
// 32^3: 617 and 478) -- without a source also where the in-place sweep's CTAs, one
// per SM at a time, nearly fill one or two waves (152 blocks of 32^3: 117 us, 123
// streamed; 304: 217 and 225).
inline bool sor_streams(const Geom& g, bool src, int n_inner, size_t es) {
  const SorRing r = SorRing::make(g, src, es);
  if (n_inner != 1 || (g.sz * es) % 16 != 0 || r.bytes() > kSorMaxSmem) return false;
  if (es == 4) return g.nx * g.ny * g.nz > 64 || g.nb > kSplitCtas;
  const int np = g.nx / 2 * g.ny, rounds = (np + r.threads - 1) / r.threads;
  const size_t whole = (size_t)(g.nx + 2) * (g.ny + 2) * (g.nz + 2) * es;
  const bool waves = !src && g.nb <= 304 && (g.nb + 56) % 152 < 57;  // 96..152 of 152
  return g.nx * g.ny * g.nz > 256 && (np >= 40 || g.nb < 1024) &&
         (whole <= kSorMaxSmem || (10 * np >= 9 * rounds * r.threads && !waves));
}
// FP32 32^3 blocks that stay staged whole, one CTA per SM, where that is one nearly
// full wave or, with two ghost layers and no source, two (form 1, us an iteration,
// vc = 1 and 2: 80 blocks 28.7 and 25.6, streamed 30.3 and 30.8; 125: 29.0, 26.6 and
// 36.6, 38.1; 304: 53.9, 52.1 and 51.9, 58.3; 64: 28.6, 25.3 and 25.3, 25.3; form 2,
// vc = 1: 80 blocks 32.9, streamed 31.3; 125: 33.0 and 37.8).
inline bool sor_staged_32(const Geom& g, bool src) {
  return (g.nb > (src && g.vc == 1 ? 114 : 76) && g.nb <= 152) ||
         (!src && g.vc == 2 && g.nb > 228 && g.nb <= 304);
}

// Kernel shapes of the fused sweep, chosen per (dtype, N, VC, scheme) by the
// autotuner (bcmg_autotune_sor) or fixed with bcmg_set_sor_variant.
enum SorVariant : int {
  SV_AUTO = 0,       // tuned choice if any, else SV_TILE_SS_256
  SV_TILE_SS_256 = 1,  // one CTA per block, source staged in shared memory
                       // (32^3: the planes streamed through it, sor_stream.cuh)
  SV_TILE_GS_256 = 2,  // one CTA per block, source read from global (L1)
  SV_TILE_SS_512 = 3,
  SV_TILE_GS_512 = 4,
  SV_PIPE_256 = 5,     // persistent, bulk-copy double buffering
  SV_PULL = 6,         // pull-form ghosts, persistent CTAs, double-buffered bulk copies
  SV_PULL_TILE = 7,    // pull-form ghosts, one CTA per block, bulk copies
  SV_COUNT = 8
};

// Red-black SOR pass(es).  fused: read A, write B with all ghosts (needs
// `push`); otherwise in place on B (A == B).
template <typename T>
cudaError_t launch_sor(const T* A, T* B, const T* s, const Geom& g, const double* coef,
                       double omega, int form, int n_inner, BlockBc bc, PushTable push,
                       bool fused, int* err, int variant, int pull_now, cudaStream_t st,
                       bool s_packed = false);
// Interior cells of every block of `src` into `dst`, N^3 per block in the
// order the pull-form SOR kernels sweep them (their packed source).
template <typename T>
cudaError_t launch_pack_source(T* dst, const T* src, const Geom& g, cudaStream_t st);
// Whether the pipelined pull-form sweeps cover this shape: cubic 8^3 / 16^3
// blocks, vc 1 or 2, two stages (tile, second field if any, 640 B of block
// constants and entries) within one CTA's shared memory.
inline bool pipe_shape_ok(int dtype_bytes, int n, int vc, bool second_field) {
  if ((n != 8 && n != 16) || (vc != 1 && vc != 2)) return false;
  const size_t lx = (size_t)n + 2 * vc, es = (size_t)dtype_bytes;
  const size_t tile = (lx * (n + 2) * (n + 2) * es + 127) / 128 * 128;
  const bool compact = (vc * lx * es) % 16 == 0;
  const size_t s = second_field ? ((size_t)n * (compact ? n * lx : lx * lx) * es + 127) / 128 * 128 : 0;
  return 2 * (tile + s + 640) <= kPipeMaxSmem;
}
inline bool sor_pull_ok(int dtype_bytes, int n, int vc, int form) {
  return pipe_shape_ok(dtype_bytes, n, vc, form == 2);
}

// Seven-point operator: per-block constants cc[b*7+c] (double, rounded to T
// in the kernel) or seven coefficient fields.
template <typename T>
struct Op {
  const double* cc;
  const T* A[7];
  const T* cf8;  // per block {Ap..At, RN(1/Ap)} rounded to T (constant operators), or null
  const T* rA0;  // coefficient fields: RN(1/Ap) per cell (launch_recip), or null
};

// Threads for ncol columns: whole warps, the last round of columns as full as
// the others.
inline int column_threads(const Geom& g) {
  const int ncol = g.nx * g.ny, rounds = (ncol + 255) / 256;
  return ((ncol + rounds - 1) / rounds + 31) / 32 * 32;
}

// Planes per CTA of the sweeps: whole blocks once they make about 16 CTAs per
// SM; fewer blocks are cut into chunks of four planes or more until they do.
inline int sweep_chunk(const Geom& g) {
  const int want = (152 * 16 + g.nb - 1) / g.nb;
  const int most = g.nz / 4 > 1 ? g.nz / 4 : 1;
  const int chunks = want < most ? want : most;
  return (g.nz + chunks - 1) / chunks;
}

// RN(1/Ap) of every interior cell of a coefficient field, 0 where the FP64
// sweeps' division by it does not apply.
cudaError_t launch_recip(double* out, const double* a, const Geom& g, cudaStream_t st);

template <typename T>
cudaError_t launch_jacobi(T* x1, const T* x0, const T* b, Op<T> op, const Geom& g, T omega,
                          cudaStream_t st);
// Fused Jacobi sweep: x1 interior, Dirichlet ghosts and pushed VC ghosts from
// x0 (per-block constant operator: cf[b*8 + 0..6] the seven coefficients and
// cf[b*8 + 7] 1/Ap, all rounded to T); every other cell of x1 (edges,
// corners, ghost layers no neighbour or Dirichlet condition writes) takes
// x0's value.  partial[b] = sum of squared residuals of x0 when partial !=
// null.  cudaErrorInvalidValue for shapes it does not cover (cubic 8/16
// blocks, vc <= 2, tiles within shared memory).  pdl: launched as a dependent of
// the kernel before (launch_dependent, bulk.cuh), which the push forms allow.
// Ghost modes of the fused sweeps.  kGhostPush: x0's ghosts are read as
// they are and the launch writes every ghost x1 feeds (x1 leaves with all
// ghosts updated).  kGhostPull: the launch first fills x0's first ghost
// layer from its neighbours' interiors and its Dirichlet ghosts (the ghost
// update that follows a sweep, done by the reader), and writes no ghost of a
// fed face -- x1's ghosts need a ghost update before anything else reads
// them.  kGhostAsIs: the pull kernel on x0's ghosts as they are (the first
// launch of a run).
// kGhostPushZero: the push form with x0 taken as zero everywhere (not read):
// the first pass of a preconditioner from zero.
// kGhostPullClose, kGhostAsIsClose: kGhostPull / kGhostAsIs (one CTA per block)
// with x1 leaving as the push form leaves it, for a run's last launch.
enum : int { kGhostPush = 0, kGhostPull = 1, kGhostAsIs = 2, kGhostPushZero = 3,
             kGhostPullClose = 4, kGhostAsIsClose = 5 };
// Kernel shapes of the pull-form Jacobi sweep: one CTA per block, or the
// persistent double-buffered pipeline.
enum : int { kJacobiTile = 1, kJacobiPipe = 2 };
// The BiCGSTAB preconditioner's zero-start pass made in one launch with the
// vector update that produces its right-hand side b: kind kPreP b = r + beta (b - gamma q) (kr_p), kPreS b = r -
// alpha q (kr_s), kPreCopy b = r; the new b is written back, the scalars
// come from the segments' records, blocks of finished segments are skipped.
enum : int { kPreNone = 0, kPreP = 1, kPreS = 2, kPreCopy = 3 };
template <typename T>
struct JacPre {
  int kind;
  const T* r;
  const T* q;
  KSegs segs;
};

template <typename T>
cudaError_t launch_jacobi_fused(const T* x0, T* x1, const T* b, const Geom& g, const T* cf,
                                T omega, BlockBc bc, PushTable push, int ghost_mode, int shape,
                                double* partial, int* err, const JacPre<T>* pre,
                                cudaStream_t st, bool pdl = false);
// mode 0: ax = A x;  mode 1: r = b - A x;  mode 2: partial[b] = sum r^2 (no store).
// streamed (residual_streams, device memory aligned to 16 bytes): the FP64 planes
// stream through shared memory, and mode 2 leaves kr_parts sums per block.  Else it
// leaves one, or sum_parts where the cubic kernels do not apply (cubic_residuals).
template <typename T>
cudaError_t launch_residual(T* out, const T* x, const T* b, Op<T> op, const Geom& g, int mode,
                            bool streamed, double* partial, int* err, cudaStream_t st);
// Per-block FP64 partial sums of x.y (interiors).
template <typename T>
cudaError_t launch_dot_partial(const T* x, const T* y, const Geom& g, double* partial,
                               cudaStream_t st);
// Sum n partials in a fixed order into *out (one CTA).
cudaError_t launch_reduce_final(const double* partial, int n, double* out, cudaStream_t st);

// Interior BLAS-1: kind 0 axpy y+=a x; 1 xpay y=x+a y; 2 axpyz z=a x+y;
// 3 axpbypz z=a x+b y+z; 4 scal z=a z.
template <typename T>
cudaError_t launch_blas1(int kind, T* z, const T* x, const T* y, T a, T b, const Geom& g,
                         cudaStream_t st);
// Folds the boundary faces of a coefficient-brick operator into its diagonal
// and the right-hand side (SolverTest bca.f90:12-394): code[b*6+f] 0 none,
// 1 Dirichlet, 2 Neumann; xc[b*6+f] the face value.  Three launches, x then
// y then z faces, so every cell sees the reference's Aw, Ae, As, An, Ab, At
// order.
template <typename T>
struct FoldPtrs {
  T* A[7];  // Ap, Aw, Ae, As, An, Ab, At
  T* b;
};
template <typename T>
cudaError_t launch_fold_boundary(FoldPtrs<T> p, const Geom& g, const int* code, const double* xc,
                                 cudaStream_t st);
// Exchange with other processes (exchange.cu): pack (values of each entry
// from its source block t.src into buf + off) or unpack (buf + off into the
// ghosts of t.dst).
template <typename T>
cudaError_t launch_xch(T* data, const Geom& g, const VcTask* ents, const int64_t* off, int n,
                       T* buf, bool pack, cudaStream_t st);

// Whether the BiCGSTAB iteration's kernels are launched as dependents of one
// another (launch_dependent, bulk.cuh): FP32 on blocks of at most 16^3, up to five
// million cells, where the gap between two launches is some per cent of a kernel (us
// an iteration without and with: 8^3, 512 blocks 57.7, 46.7; 2197 77.2, 66.1; 5152
// 144, 126; 12^3, 1000 blocks 138, 122; 16^3, 64 blocks 67.7, 57.1; 1000 162.5, 160.1).
// Not 16^3 in between: a waiting CTA of its streamed A.x holds shared memory that the
// kernel before could use (216 blocks 78.5, 83.7; 512 98.8, 104.7; 729 123, 126).  Not
// on larger meshes: 1427 blocks of 16^3 276 and 281, 2549 419 and 447; and a
// dependent's waiting CTAs hold slots that other streams' kernels would take (200
// served requests on four streams: median latency 8 s without, 12 s with, 5.88 and
// 5.82 solves a second).  Nor in FP64 (342 blocks of 32^3: 38.6 ms without, 40.7).
inline bool kr_dependent(size_t es, const Geom& g) {
  const int cells = g.nx * g.ny * g.nz;
  if (es != 4 || cells > 4096 || (int64_t)g.nb * cells > 8 * 152 * 4096) return false;
  return !(g.nx == 16 && g.ny == 16 && g.nz == 16) || g.nb <= 152 || g.nb >= 800;
}

// Parts of a block's planes that the kernels with inner products take as CTAs of
// their own in FP64 and for coefficient fields: two thousand cells or more and
// four planes, at most four parts.  They are bound by the FP64 pipe (or by the
// bytes in flight), so a mesh of a few hundred blocks should not leave an SM with
// three blocks beside one with two.  The parts' sums are added in order, and the
// split depends on the block's shape alone: a system's sums are the same alone
// and among others.
inline int kr_parts(const Geom& g) {
  const int by_cells = g.nx * g.ny * g.nz / 2048, by_planes = g.nz / 4;
  const int n = by_cells < by_planes ? by_cells : by_planes;
  return n < 1 ? 1 : n > 4 ? 4 : n;
}
constexpr int kKrMaxParts = 4;
// Parts per block of calc_r2 on blocks of any shape and coefficient fields, a
// partial sum each.  A CTA a block left few blocks to walk alone: 64 blocks of
// 28^3, FP64 fields, 220 us, in four parts 60 (fields read plane by plane, 160);
// 288 of 32^3, FP32, 130 and 86.  FP64 gains at every count (1408 of 28^3: 1027 and
// 932), and so do blocks of four parts in FP32 (267 and 252); smaller ones lose in
// FP32 from four CTAs an SM on (512 of 16^3: 17 us, in two parts 19).
inline int sum_parts(const Geom& g, size_t es) {
  const int most = kr_parts(g);
  if (es == 8 || most == kKrMaxParts) return most;
  int n = 1;
  while (n < most && g.nb * (n + 1) <= kSplitCtas) n++;
  return n;
}
// Whether calc_ax / calc_r / calc_r2 have the kernels of cubic blocks with a
// constant operator.
inline bool cubic_residuals(bool constant_op, const Geom& g) {
  return constant_op && g.nx == g.ny && g.ny == g.nz && (g.vc == 1 || g.vc == 2) &&
         (g.nx == 8 || g.nx == 16 || g.nx == 32);
}
inline bool residual_streams(size_t es, bool constant_op, const Geom& g) {
  return es == 8 && constant_op && g.nx == g.ny && g.ny == g.nz && (g.nx == 16 || g.nx == 32) &&
         (g.vc == 1 || g.vc == 2);
}

// Device-resident BiCGSTAB iteration (krylov.cu): see krylov.cuh.
template <typename T>
cudaError_t launch_kr_p(T* p, const T* r, const T* q, const Geom& g, KSegs S, cudaStream_t st);
template <typename T>
cudaError_t launch_kr_s(T* s, const T* r, const T* q, const Geom& g, KSegs S, cudaStream_t st);
// parts: partial sums per block (1 or kr_parts), part p of block b at
// partial[b * parts + p], the second sums nb * parts further on.
template <typename T>
cudaError_t launch_kr_ax(T* out, const T* x, Op<T> op, const T* y0, int ndot, const Geom& g,
                         int parts, KSegs S, double* partial, int* err, cudaStream_t st);
template <typename T>
cudaError_t launch_kr_xr(T* x, T* r, const T* p_, const T* s_, const T* s, const T* t,
                         const T* r0, const Geom& g, int parts, KSegs S, double* partial, int* err,
                         cudaStream_t st);
// A preconditioner's pass from x0 = 0 on blocks of any shape or coefficient
// fields: x1's interior from b, or from b made of the BiCGSTAB vectors (pre).
template <typename T>
cudaError_t launch_kr_zero_pass(T* x1, T* b, const JacPre<T>& pre, const Op<T>& op, const Geom& g,
                                T omega, cudaStream_t st);
template <typename T>
cudaError_t launch_kr_dot2(const T* x, const T* y, const T* u, const T* v, const Geom& g,
                           double* partial, cudaStream_t st);
template <typename T>
cudaError_t launch_kr_best(T* xbest, const T* x, const Geom& g, KSegs S, cudaStream_t st);
cudaError_t launch_kr_scalar(const double* partial, int nb, int parts, KSegs S, int stage,
                             int max_iter, double eps2, int keep_best, bool dependent,
                             cudaStream_t st);
cudaError_t launch_kr_segsum(const double* partial, int nb, KSegs S, double* out,
                             cudaStream_t st);
template <typename T>
cudaError_t launch_kr_seg_copy(T* dst, const T* src, const Geom& g, const int* seg_of,
                               const unsigned char* flag, cudaStream_t st);
cudaError_t launch_kr_seg_to32(float* r32, const double* r64, const Geom& g32, const Geom& g64,
                               const int* seg_of, const unsigned char* flag, const double* scale,
                               cudaStream_t st);
cudaError_t launch_kr_seg_acc(double* x64, const float* d32, const Geom& g32, const Geom& g64,
                              const int* seg_of, const unsigned char* flag, const double* scale,
                              cudaStream_t st);

// The cells of every brick that the pull-form sweeps never write, dst <- src:
// the ghost planes in z and, with `rows`, the ghost rows in y of the others.
template <typename T>
cudaError_t launch_copy_frame(T* dst, const T* src, const Geom& g, bool rows, cudaStream_t st);

template <typename T>
cudaError_t launch_fill(T* x, int64_t n, T v, cudaStream_t st);
template <typename T>
cudaError_t launch_fill_random(T* x, const Geom& g, int b0, int nb, uint64_t seed, double lo,
                               double hi, cudaStream_t st);

}  // namespace bcmg
