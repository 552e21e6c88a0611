// Multigrid-preconditioned CG for the pressure Poisson problem
// (linsolve/poisson_solver.cpp:678-809) on compact, ghost-free vectors.
//
// Algorithm: the reference's exactly -- PCG on A = -Lap_h with BC-aware
// neighbours (:195-269), one V(2,2) cycle per iteration with damped Jacobi
// (omega = 2/3), 2x2x2 cell-average restriction, piecewise-constant
// prolongation and a dense partially-pivoted Gaussian elimination on the
// coarsest grid, and the zero-mean projection on singular (periodic /
// all-Neumann) problems after every update.
//
// B200 form: an iteration passes over the fine level's vectors four times
// (march.cuh): k_descend, k_ascend, k_direction and k_advance, each several
// steps of the algorithm pipelined over the planes of a tile, with the sums the
// next one needs (deterministic two-stage reduction, common.cuh).  The coarse
// levels take the same two V-cycle kernels each, down to the level that is one
// matrix.  A mean removal is never a separate pass: the kernel that produces
// a vector records its mean as a pending shift that consumers subtract on load.
// The V-cycle storage type T is double (OF_FP64) or float (OF_MIXED: FP32
// storage and arithmetic inside an FP64 defect correction).
#include "kernels.hpp"
#include "march.cuh"

#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <memory>
#include <type_traits>
#include <vector>

namespace ofb {

namespace {

constexpr double kSmallNumber = 1.0e-30;
constexpr double kOmega = 2.0 / 3.0;
constexpr int kMaxCoarse = 1024;

template <int K>
__device__ __forceinline__ void zero(double (&v)[K]) {
#pragma unroll
  for(int q = 0; q < K; ++q) v[q] = 0.0;
}

#define STENCIL_PROLOGUE(L)                                 \
  const int i = blockIdx.x * kTX + threadIdx.x;             \
  const int j = blockIdx.y * kTY + threadIdx.y;             \
  const bool valid = i < (L).nx && j < (L).ny;              \
  const int k0 = blockIdx.z * kchunk;                       \
  const int k1 = min(k0 + kchunk, (L).nz);

// ---------------------------------------------------------------------------
// The small end of the hierarchy as one matrix.  From the first level of at
// most kDenseCells cells down to the coarsest, v_cycle (:597-633) is a fixed
// linear map of that level's rhs (sweeps, restriction, elimination and mean
// removals are all linear), so its matrix G is formed once per plan -- column
// c is the V-cycle of the unit vector e_c, one block each (k_dense_columns) --
// and a solve applies it with one matrix-vector product (k_dense_apply).
//
// Replaying the V-cycle instead costs one block ~45 barrier-separated phases,
// and above 32 coarse unknowns an elimination of two barriers per unknown:
// 27 us per V-cycle from 16^3 down, 207 us with 135 coarse unknowns (96 x 80 x
// 72), 578 us with 315 (144 x 80 x 112).  G of 512 cells is 2 MB and of 1024
// cells 8 MB, read from L2 by a block per kDenseRows rows in a few us; above
// 1024 cells it would leave L2 no room (4096 cells: 134 MB).
// ---------------------------------------------------------------------------
constexpr int kDenseCells = 1024;
constexpr int kTailMaxLevels = 12;
constexpr int kTailThreads = 512;

// Per tail level (all but the coarsest), built on the host when the plan is
// made and staged into shared memory by every block of k_dense_columns:
//   nbr[6][n]   the six operand positions of each cell under the boundary
//               rules (nb_lo / nb_hi: neighbour, periodic image, or the cell
//               itself), as +-(index + 1), minus for a homogeneous-Dirichlet
//               image (ghost = -centre); order x-, x+, y-, y+, z-, z+
//   parent[n]   the cell's parent on the next coarser level
//   child[nc][nch]  each coarser cell's children in dz, dy, dx order
//   cls[n]      the cell's boundary class (x + 4 y + 16 z, each 0 interior,
//               1 first, 2 last, 3 both) and
//   itab[64]    the Jacobi inverse diagonal of each class (T)
// so a tail phase does no index arithmetic and reads no boundary flags.
struct TailLevel {
  OpInfo op;
  int off;         // offset of the level's b, x, s arrays in shared memory (elements)
  int tab;         // byte offset of the level's tables in the table region
  int nch;         // children per coarser cell
};

struct TailArgs {
  int count;  // levels in the tail; the last one is the coarsest
  TailLevel lv[kTailMaxLevels];
  int coarse_n;
  int coarse_off;  // offset (elements, 8-byte aligned) of the FP64 solve vector
  int fact_off;    // offset (8-byte aligned) of the staged factors (coarse_n <= 32)
  int tab_off;     // byte offset (16-aligned) of the table region in shared memory
  int tab_bytes;   // its size (a multiple of 16)
  const unsigned char* tabs;  // the tables in device memory
  const int* swaps;
  const double* factors;
  int zm;
};

// Byte layout of one tail level's tables (see TailLevel).
struct TailTabLayout {
  size_t nbr, parent, child, cls, itab, bytes;
};

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) / 16 * 16; }

__host__ __device__ inline TailTabLayout tail_tab_layout(int n, int nc, int nch, size_t tsz) {
  TailTabLayout t;
  t.nbr = 0;
  t.parent = 12 * static_cast<size_t>(n);
  t.child = t.parent + 2 * static_cast<size_t>(n);
  t.cls = t.child + 2 * static_cast<size_t>(nc) * nch;
  t.itab = align16(t.cls + static_cast<size_t>(n));
  t.bytes = align16(t.itab + 64 * tsz);
  return t;
}

// Block-wide sum; every thread gets the same total (fixed order).  red has
// 33 entries: the warp partials and the total.
__device__ __forceinline__ double tail_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(lane == 0) red[warp] = v;
  __syncthreads();
  if(warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    double x = lane < nw ? red[lane] : 0.0;
    x = warp_sum(x);
    if(lane == 0) red[32] = x;
  }
  __syncthreads();
  return red[32];
}

// Ends a tail phase: the block barrier, with the block-wide sum of v (warp
// partials alternate between two rows of red so that a fast thread's next
// phase never overwrites partials a slow thread is still adding).
__device__ __forceinline__ double tail_phase_sum(double v, double (*red)[32], int& par) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(lane == 0) red[par][warp] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  double t = 0.0;
  for(int w = 0; w < nw; ++w) t += red[par][w];
  par ^= 1;
  return t;
}

// One operand value through a table entry e = +-(index + 1).
template <typename A, typename Op>
__device__ __forceinline__ A tab_nb(int e, Op op) {
  const A v = op(e < 0 ? -e - 1 : e - 1);
  return e < 0 ? -v : v;
}

// A u at cell q from the staged neighbour table; c gets u at q.
template <typename A, typename Op>
__device__ __forceinline__ A tab_apply(const short* nbr, int n, int q, A ix, A iy, A iz, Op op, A& c) {
  c = op(q);
  const A l = tab_nb<A>(nbr[q], op);
  const A r = tab_nb<A>(nbr[n + q], op);
  const A d = tab_nb<A>(nbr[2 * n + q], op);
  const A u = tab_nb<A>(nbr[3 * n + q], op);
  const A b = tab_nb<A>(nbr[4 * n + q], op);
  const A f = tab_nb<A>(nbr[5 * n + q], op);
  const A two_c = A(2) * c;
  return -(r - two_c + l) * ix - (u - two_c + d) * iy - (f - two_c + b) * iz;
}

// The tail V-cycle of the unit vector e_c (its mean removed on singular
// problems, as the rhs of every level has it removed) in the calling block;
// x_out gets the result, its mean removed.  sm is the tail's shared-memory
// layout (TailArgs).
template <typename T>
__device__ void vcycle_tail_column(const TailArgs& a, int c, T* __restrict__ x_out, double* sm) {
  using A = double;
  __shared__ double red[2][32];
  int par = 0;
  const int tid = threadIdx.x, bd = blockDim.x;
  const int zm = a.zm;
  const A om = A(kOmega);
  auto B = [&](int l) { return sm + a.lv[l].off; };
  auto X = [&](int l) { return sm + a.lv[l].off + a.lv[l].op.L.count(); };
  auto S = [&](int l) { return sm + a.lv[l].off + 2 * a.lv[l].op.L.count(); };
  unsigned char* tabs = reinterpret_cast<unsigned char*>(sm) + a.tab_off;
  const int last = a.count - 1;
  const int nco = a.coarse_n;
  double* fact = reinterpret_cast<double*>(sm + a.fact_off);
  int* swp = reinterpret_cast<int*>(fact + (nco <= 32 ? nco * nco : 0));
  if(nco <= 32) {
    // the coarse factors, read by the one-warp elimination below
    for(int q = tid; q < nco * nco; q += bd) fact[q] = a.factors[q];
    for(int q = tid; q < nco; q += bd) swp[q] = a.swaps[q];
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.tabs);
    uint4* dst = reinterpret_cast<uint4*>(tabs);
    for(int q = tid; q < a.tab_bytes / 16; q += bd) dst[q] = __ldg(&src[q]);
    const int n0 = a.lv[0].op.L.count();
    const double mean = zm ? 1.0 / n0 : 0.0;
    for(int q = tid; q < n0; q += bd) B(0)[q] = (q == c ? 1.0 : 0.0) - mean;
  }
  __syncthreads();
  double sbs[kTailMaxLevels], sxs[kTailMaxLevels];
  sbs[0] = 0.0;
  // descent
  for(int l = 0; l < last; ++l) {
    const TailLevel& tl = a.lv[l];
    const int n = tl.op.L.count();
    const int nc = a.lv[l + 1].op.L.count();
    const TailTabLayout lay = tail_tab_layout(n, nc, tl.nch, sizeof(double));
    const short* nbr = reinterpret_cast<const short*>(tabs + tl.tab + lay.nbr);
    const short* child = reinterpret_cast<const short*>(tabs + tl.tab + lay.child);
    const unsigned char* cls = tabs + tl.tab + lay.cls;
    const A* itab = reinterpret_cast<const A*>(tabs + tl.tab + lay.itab);
    auto dinv = [&](int p) { return itab[cls[p]]; };
    const A ix = A(tl.op.inv2[0]), iy = A(tl.op.inv2[1]), iz = A(tl.op.inv2[2]);
    auto apply = [&](int q, auto op, A& c) { return tab_apply<A>(nbr, n, q, ix, iy, iz, op, c); };
    const A* b = B(l);
    A* x = X(l);
    A* s = S(l);
    const A sbl = A(sbs[l]);
    // both pre-sweeps from a zero correction
    double part = 0.0;
    for(int q = tid; q < n; q += bd) {
      A c;
      const A ax = apply(q, [&](int p) { return om * (b[p] - sbl) * dinv(p); }, c);
      const A v = c + om * ((b[q] - sbl) - ax) * dinv(q);
      x[q] = v;
      part += double(v);
    }
    {
      const double t = tail_phase_sum(part, red, par);
      sxs[l] = zm ? t / n : 0.0;
    }
    // residual (b - sb) - A (x - sx)
    const A sxl = A(sxs[l]);
    for(int q = tid; q < n; q += bd) {
      A c;
      const A ax = apply(q, [&](int p) { return x[p] - sxl; }, c);
      s[q] = (b[q] - sbl) - ax;
    }
    __syncthreads();
    // restrict_full_weighting (:397-424), children in dz, dy, dx order
    const int nch = tl.nch;
    const A inv_children = A(1.0 / double(nch));
    A* bc = B(l + 1);
    part = 0.0;
    for(int Q = tid; Q < nc; Q += bd) {
      A sum = A(0);
      for(int t = 0; t < nch; ++t) sum += s[child[Q * nch + t]];
      const A v = inv_children * sum;
      bc[Q] = v;
      part += double(v);
    }
    {
      const double t = tail_phase_sum(part, red, par);
      sbs[l + 1] = zm ? t / nc : 0.0;
    }
  }
  // direct_coarse_solve (:530-567): the host elimination replayed on the rhs
  // (its mean removed first, as the reference does before the solve).  Up to
  // 32 unknowns (every grid the hierarchy coarsens to 2 per axis) one warp
  // replays it with the rhs in registers and the factors in shared memory,
  // the same operations in the same order as the block-wide form below.
  if(nco <= 32) {
    const int n = nco;
    if(tid < 32) {
      constexpr unsigned kFull = 0xffffffffu;
      const int lane = tid;
      double yv = lane < n ? double(B(last)[lane]) - sbs[last] : 0.0;
      if(zm && lane == n - 1) yv = 0.0;
      for(int p = 0; p < n; ++p) {
        const int sp = swp[p];
        if(sp != p) {
          const double at_p = __shfl_sync(kFull, yv, p);
          const double at_s = __shfl_sync(kFull, yv, sp);
          if(lane == p) yv = at_s;
          else if(lane == sp) yv = at_p;
        }
        const double yp = __shfl_sync(kFull, yv, p);
        if(lane > p && lane < n) {
          const double factor = fact[lane * n + p];
          if(factor != 0.0) yv -= factor * yp;
        }
      }
      for(int row = n - 1; row >= 0; --row) {
        if(lane == row) yv = yv / fact[row * n + row];
        const double yr = __shfl_sync(kFull, yv, row);
        if(lane < row) yv -= fact[lane * n + row] * yr;
      }
      const double sum = __shfl_sync(kFull, warp_sum(lane < n ? yv : 0.0), 0);
      const double mean = zm ? sum / n : 0.0;
      if(lane < n) X(last)[lane] = A(yv - mean);
    }
    __syncthreads();
  } else {
    const int n = nco;
    __shared__ double cred[33];
    A* y = B(last);
    A* xc = X(last);
    double* yd = reinterpret_cast<double*>(sm + a.coarse_off);  // solve in FP64
    for(int q = tid; q < n; q += bd) yd[q] = double(y[q]) - sbs[last];
    __syncthreads();
    if(zm && tid == 0) yd[n - 1] = 0.0;
    __syncthreads();
    for(int p = 0; p < n; ++p) {
      if(tid == 0 && a.swaps[p] != p) {
        const double tmp = yd[p];
        yd[p] = yd[a.swaps[p]];
        yd[a.swaps[p]] = tmp;
      }
      __syncthreads();
      const double yp = yd[p];
      for(int r = p + 1 + tid; r < n; r += bd) {
        const double factor = a.factors[static_cast<size_t>(r) * n + p];
        if(factor != 0.0) yd[r] -= factor * yp;
      }
      __syncthreads();
    }
    for(int row = n - 1; row >= 0; --row) {
      if(tid == 0) yd[row] = yd[row] / a.factors[static_cast<size_t>(row) * n + row];
      __syncthreads();
      const double yr = yd[row];
      for(int r = tid; r < row; r += bd) yd[r] -= a.factors[static_cast<size_t>(r) * n + row] * yr;
      __syncthreads();
    }
    double part = 0.0;
    for(int q = tid; q < n; q += bd) part += yd[q];
    const double sum = tail_sum(part, cred);
    const double mean = zm ? sum / n : 0.0;
    for(int q = tid; q < n; q += bd) xc[q] = A(yd[q] - mean);
    __syncthreads();
  }
  // ascent: prolongate_and_add (:426-451) + first post-sweep, second post-sweep
  double sxc = 0.0;  // the coarse correction has its mean removed
  for(int l = last - 1; l >= 0; --l) {
    const TailLevel& tl = a.lv[l];
    const int n = tl.op.L.count();
    const int nc = a.lv[l + 1].op.L.count();
    const TailTabLayout lay = tail_tab_layout(n, nc, tl.nch, sizeof(double));
    const short* nbr = reinterpret_cast<const short*>(tabs + tl.tab + lay.nbr);
    const short* parent = reinterpret_cast<const short*>(tabs + tl.tab + lay.parent);
    const unsigned char* cls = tabs + tl.tab + lay.cls;
    const A* itab = reinterpret_cast<const A*>(tabs + tl.tab + lay.itab);
    auto dinv = [&](int p) { return itab[cls[p]]; };
    auto parent_of = [&](int p) { return static_cast<int>(parent[p]); };
    const A ix = A(tl.op.inv2[0]), iy = A(tl.op.inv2[1]), iz = A(tl.op.inv2[2]);
    auto apply = [&](int q, auto op, A& c) { return tab_apply<A>(nbr, n, q, ix, iy, iz, op, c); };
    const A* b = B(l);
    A* x = X(l);
    A* s = S(l);
    const A* xc = X(l + 1);
    const A sbl = A(sbs[l]), sxl = A(sxs[l]), sec = A(sxc);
    double part = 0.0;
    for(int q = tid; q < n; q += bd) {
      A c;
      const A ax = apply(q, [&](int p) { return (x[p] - sxl) + (xc[parent_of(p)] - sec); }, c);
      const A v = c + om * ((b[q] - sbl) - ax) * dinv(q);
      s[q] = v;
      part += double(v);
    }
    double sa;
    {
      const double t = tail_phase_sum(part, red, par);
      sa = zm ? t / n : 0.0;
    }
    const A saa = A(sa);
    part = 0.0;
    for(int q = tid; q < n; q += bd) {
      A c;
      const A ax = apply(q, [&](int p) { return s[p] - saa; }, c);
      const A v = c + om * ((b[q] - sbl) - ax) * dinv(q);
      x[q] = v;
      part += double(v);
    }
    {
      const double t = tail_phase_sum(part, red, par);
      sxc = zm ? t / n : 0.0;
    }
  }
  const int n0 = a.lv[0].op.L.count();
  const A s0 = A(sxc);
  for(int q = tid; q < n0; q += bd) x_out[q] = T(X(0)[q] - s0);
}

// Column c of G, one block per column: G[c * n + row] (FP32 on the mixed path,
// formed in FP64).
template <typename T>
__global__ void __launch_bounds__(kTailThreads) k_dense_columns(TailArgs a, T* __restrict__ G) {
  extern __shared__ __align__(16) unsigned char tail_smem[];
  const int n = a.lv[0].op.L.count();
  vcycle_tail_column<T>(a, blockIdx.x, G + static_cast<size_t>(blockIdx.x) * n,
                        reinterpret_cast<double*>(tail_smem));
}

// x = G b, sums in FP64.  A block owns kDenseRows rows; its threads split the
// columns into groups, so that a warp reads runs of kDenseRows consecutive
// entries of a column (128 bytes in FP64) and every thread has the loads of
// its n / 16 columns in flight at once; the groups' partial sums meet in shared
// memory in a fixed order.  Bound by the read of G from L2 (n = 512: 2 MB over
// 32 blocks).  G removes the rhs's and the result's mean, so no shift is read
// or left.  With sc (the dense level is the finest) it also forms r.z.
constexpr int kDenseRows = 16;
constexpr int kDenseThreads = 256;

template <typename T, typename B>
__global__ void __launch_bounds__(kDenseThreads)
    k_dense_apply(int n, const T* __restrict__ G, const B* __restrict__ b, T* __restrict__ x,
                  LevelScalars* ls, SolveScalars* sc, RedBuf rb) {
  pdl_early();
  pdl_enter();
  constexpr int kGroups = kDenseThreads / kDenseRows;
  __shared__ double part[kGroups][kDenseRows + 1];
  __shared__ double bs[kDenseCells];
  const int r = threadIdx.x % kDenseRows, grp = threadIdx.x / kDenseRows;
  const int row = blockIdx.x * kDenseRows + r;
  for(int q = threadIdx.x; q < n; q += kDenseThreads) bs[q] = double(b[q]);
  __syncthreads();
  double sum = 0.0;
  if(row < n) {
#pragma unroll 8
    for(int c = grp; c < n; c += kGroups) sum += double(__ldg(&G[static_cast<size_t>(c) * n + row])) * bs[c];
  }
  part[grp][r] = sum;
  __syncthreads();
  double acc[2] = {0.0, 0.0};
  if(grp == 0 && row < n) {
    double v = 0.0;
#pragma unroll
    for(int k = 0; k < kGroups; ++k) v += part[k][r];
    x[row] = T(v);
    acc[0] = double(T(v));
    acc[1] = bs[row] * double(T(v));
  }
  if(sc == nullptr) {
    if(blockIdx.x == 0 && threadIdx.x == 0) ls->sx = 0.0;  // the mean is already removed
    return;
  }
  const bool mx[2] = {false, false};
  reduce_finish<2>(acc, mx, rb, [=](const Sums<2>& s) {
    const double mean = sc->zero_mean ? s.v[0] / n : 0.0;
    ls->sx = mean;
    // r.z with z = x - mean, r = b - sr (linsolve/poisson_solver.cpp:749, :791)
    const double rz_new = s.v[1] - mean * (sc->sum_r - sc->n * sc->sr) - sc->sr * s.v[0];
    if(!sc->first) sc->beta = rz_new / sc->rz;
    sc->rz = rz_new;
  });
}

// ---------------------------------------------------------------------------
// CG kernels (FP64 vectors).
// ---------------------------------------------------------------------------

// A solve from a zero guess: r = b - sb, x = 0 and the solve's scalars, in one
// flat pass (1 vector read, 2 written; clearing x and the general residual
// took 21 + 125 us at 256^3).
constexpr int kFlatThreads = 256, kFlatUnroll = 4;

__global__ void __launch_bounds__(kFlatThreads)
    k_start_from_zero(int n, const double* __restrict__ b, double* __restrict__ x, double* __restrict__ r,
                      SolveScalars* sc, march::SolveStart start, RedBuf rb) {
  const double sb = start.zero_mean ? sc->sb : 0.0;
  const int stride = gridDim.x * blockDim.x;
  double acc[2] = {0.0, 0.0};
  for(int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += kFlatUnroll * stride) {
    double v[kFlatUnroll];
#pragma unroll
    for(int u = 0; u < kFlatUnroll; ++u) v[u] = q + u * stride < n ? b[q + u * stride] - sb : 0.0;
#pragma unroll
    for(int u = 0; u < kFlatUnroll; ++u)
      if(q + u * stride < n) {
        r[q + u * stride] = v[u];
        x[q + u * stride] = 0.0;
        acc[0] += v[u];
        acc[1] += v[u] * v[u];
      }
  }
  const bool mx[2] = {false, false};
  reduce_finish<2>(acc, mx, rb, [=](const Sums<2>& s) {
    sc->sx = 0.0;
    march::start_solve(sc, start, s.v[0], s.v[1]);
  });
}

// First node of the loop graph: run the body at all?
__global__ void k_loop_gate(const SolveScalars* sc, cudaGraphConditionalHandle cond) {
  cudaGraphSetConditional(cond, sc->cont);
}

// Mixed path: the FP64 residual scaled to unit RMS into the FP32 inner rhs,
// the inner correction cleared, and the inner loop's scalars initialised as
// start_solve (march.cuh) does it for a zero initial guess.
__global__ void __launch_bounds__(kTX* kTY)
    k_dc_to_inner(CLay L, const double* __restrict__ r, const SolveScalars* sc,
                  float* __restrict__ r32, float* __restrict__ e32, SolveScalars* si, double inner_tol,
                  int inner_max_it, int kchunk, RedBuf rb, cudaGraphConditionalHandle cond) {
  STENCIL_PROLOGUE(L)
  const double sr = sc->sr;
  const double inv = sc->rnorm > 0.0 ? 1.0 / sc->rnorm : 1.0;
  double acc[2];
  zero(acc);
  if(valid) {
    for(int k = k0; k < k1; ++k) {
      const int q = L.idx(i, j, k);
      const float v = float((r[q] - sr) * inv);
      r32[q] = v;
      e32[q] = 0.0f;
      acc[0] += double(v);
      acc[1] += double(v) * double(v);
    }
  }
  const bool mx[2] = {false, false};
  reduce_finish<2>(acc, mx, rb, [=](const Sums<2>& s) {
    const int n = sc->n;
    si->n = n;
    si->zero_mean = sc->zero_mean;
    si->tol = inner_tol;
    si->max_it = inner_max_it;
    const double srn = si->zero_mean ? s.v[0] / n : 0.0;
    si->sr = srn;
    si->sum_r = s.v[0];
    const double r0 = sqrt(fmax(s.v[1] - n * srn * srn, 0.0) / n);
    si->r0 = r0;
    si->rnorm = r0;
    si->rel = 1.0;
    si->iterations = 0;
    si->stop = 0;
    si->converged = 0;
    si->first = 1;
    si->body_runs = 0;
    si->sx = 0.0;
    si->hist = nullptr;
    si->hist_cap = 0;
    si->cont = r0 > 0.0 ? 1 : 0;
    if(cond) cudaGraphSetConditional(cond, si->cont);
  });
}

// Mixed path: x = (x - sx) + scale (e - sx_inner) with the scale the inner
// rhs was divided by; records mean(x).
__global__ void __launch_bounds__(kTX* kTY)
    k_dc_update_x(CLay L, double* __restrict__ x, const float* __restrict__ e32, SolveScalars* sc,
                  const SolveScalars* si, int kchunk, RedBuf rb) {
  STENCIL_PROLOGUE(L)
  const double scale = sc->rnorm > 0.0 ? sc->rnorm : 1.0;
  const double sx = sc->sx, sxi = si->sx;
  double acc[1];
  zero(acc);
  if(valid) {
    for(int k = k0; k < k1; ++k) {
      const int q = L.idx(i, j, k);
      const double v = (x[q] - sx) + scale * (double(e32[q]) - sxi);
      x[q] = v;
      acc[0] += v;
    }
  }
  const bool mx[1] = {false};
  reduce_finish<1>(acc, mx, rb, [=](const Sums<1>& s) {
    sc->sx = sc->zero_mean ? s.v[0] / sc->n : 0.0;
  });
}

__global__ void k_compact_to_pressure(Grid g, const double* __restrict__ x, const SolveScalars* sc,
                                      double* __restrict__ p) {
  const Lay P = make_lay(g, kCell);
  const CLay L = make_clay(g.nx, g.ny, g.nz);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if(i >= L.nx || j >= L.ny) return;
  p[P.idx(i + 1, j + 1, k + 1)] = x[L.idx(i, j, k)] - sc->sx;
}

}  // namespace

// ---------------------------------------------------------------------------
// Plan
// ---------------------------------------------------------------------------

struct Level {
  Grid g;
  CLay L;
  OpInfo op;
  void* a = nullptr;   // smoother output a
  void* x = nullptr;   // smoother output b (correction)
  void* b = nullptr;   // rhs (levels >= 1)
  double* invd = nullptr;
  int rx = 1, ry = 1, rz = 1;  // refinement ratio to the next coarser level
  march::Tile tile{};          // of k_descend and k_ascend
  dim3 tgrid;
};

struct PoissonPlan {
  Grid g;
  PBC pbc;
  int precision = 0;
  int zero_mean = 1;
  std::vector<Level> levels;
  int coarse_n = 0;
  LevelScalars* ls = nullptr;  // device, one per level
  double *b = nullptr, *x = nullptr, *r = nullptr, *p = nullptr;
  double* hist = nullptr;
  int hist_cap = 0;
  size_t bytes = 0;
  // the whole solve as one CUDA graph (built on first use)
  bool use_graph = true;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  long long pre_counts[kKernelCount] = {};
  long long body_counts[kKernelCount] = {};
  // mixed path: inner (FP32) CG vectors and scalars
  float *r32 = nullptr, *e32 = nullptr, *p32 = nullptr;
  SolveScalars* sc_in = nullptr;
  int sms = 148;         // streaming multiprocessors of the plan's device
  bool all_periodic = false;  // every face periodic: constant diagonal, no boundary signs
  march::Tile cg_tile{}, res_tile{};  // of k_direction and k_advance; of k_residual
  dim3 cg_grid, res_grid;
  double* p2 = nullptr;     // second p buffer
  float* p32b = nullptr;
  // levels tail_first.. run as one matrix-vector product (k_dense_apply)
  int tail_first = -1;
  void* dense = nullptr;  // their V-cycle's matrix, column by column
  size_t dense_bytes = 0;
};

namespace {

bool can_coarsen_axis(int cells) { return cells > 1 && cells % 2 == 0 && cells > 2; }

OpInfo make_op(const Grid& g, const PBC& pbc) {
  OpInfo o;
  o.L = make_clay(g.nx, g.ny, g.nz);
  for(int a = 0; a < 3; ++a) {
    const double h = g.h(a);
    o.inv2[a] = 1.0 / (h * h);
    o.periodic[a] = pbc.type[2 * a] == kPPeriodic ? 1 : 0;
    o.dir_lo[a] = pbc.type[2 * a] == kPDirichlet ? 1 : 0;
    o.dir_hi[a] = pbc.type[2 * a + 1] == kPDirichlet ? 1 : 0;
  }
  o.invd = nullptr;
  return o;
}

// compute_operator_diagonal (linsolve/poisson_solver.cpp:271-314) by boundary class.
std::vector<double> inverse_diagonal_table(const Grid& g, const PBC& pbc) {
  std::vector<double> t(64, 0.0);
  for(int cz = 0; cz < 4; ++cz)
    for(int cy = 0; cy < 4; ++cy)
      for(int cx = 0; cx < 4; ++cx) {
        const int cls[3] = {cx, cy, cz};
        double value = 0.0;
        for(int a = 0; a < 3; ++a) {
          const double inv = 1.0 / std::pow(g.h(a), 2.0);
          double coefficient = 2.0 * inv;
          if(pbc.type[2 * a] == kPPeriodic) {
            value += coefficient;
            continue;
          }
          const bool first = cls[a] == 1 || cls[a] == 3;
          const bool last = cls[a] == 2 || cls[a] == 3;
          if(first) coefficient += pbc.type[2 * a] == kPDirichlet ? inv : -inv;
          if(last) coefficient += pbc.type[2 * a + 1] == kPDirichlet ? inv : -inv;
          value += coefficient;
        }
        t[cx + 4 * cy + 16 * cz] = value != 0.0 ? 1.0 / value : 0.0;
      }
  return t;
}

// Device memory of the plan's setup, freed with its scope.
struct DeviceBytes {
  void* p = nullptr;
  explicit DeviceBytes(size_t n) {
    if(n > 0) OFB_CHECK(cudaMalloc(&p, n));
  }
  ~DeviceBytes() { cudaFree(p); }
  DeviceBytes(const DeviceBytes&) = delete;
  DeviceBytes& operator=(const DeviceBytes&) = delete;
};

// Host copy of apply_poisson_operator with homogeneous rules, for assembling
// the coarse matrix column by column as direct_coarse_solve does.
void host_apply(const Grid& g, const PBC& pbc, const std::vector<double>& in,
                std::vector<double>& out) {
  const CLay L = make_clay(g.nx, g.ny, g.nz);
  auto val = [&](int i, int j, int k) { return in[L.idx(i, j, k)]; };
  for(int k = 0; k < L.nz; ++k)
    for(int j = 0; j < L.ny; ++j)
      for(int i = 0; i < L.nx; ++i) {
        const double c = val(i, j, k);
        const int pos[3] = {i, j, k};
        double nb[3][2];
        for(int a = 0; a < 3; ++a) {
          for(int s = 0; s < 2; ++s) {
            int q[3] = {i, j, k};
            const bool upper = s == 1;
            const int n = L.n(a);
            if((!upper && pos[a] > 0) || (upper && pos[a] < n - 1)) {
              q[a] += upper ? 1 : -1;
              nb[a][s] = val(q[0], q[1], q[2]);
              continue;
            }
            const int type = pbc.type[2 * a + s];
            if(type == kPPeriodic) {
              q[a] = upper ? 0 : n - 1;
              nb[a][s] = val(q[0], q[1], q[2]);
            } else if(type == kPNeumann) {
              nb[a][s] = c;
            } else {
              nb[a][s] = -c;
            }
          }
        }
        out[L.idx(i, j, k)] = -(nb[0][1] - 2.0 * c + nb[0][0]) / (g.dx * g.dx) -
                              (nb[1][1] - 2.0 * c + nb[1][0]) / (g.dy * g.dy) -
                              (nb[2][1] - 2.0 * c + nb[2][0]) / (g.dz * g.dz);
      }
}

}  // namespace

namespace {

// Chooses the first level of at most kDenseCells cells (the coarsest has no
// more, so there is one), lays out the shared memory of its V-cycle -- per
// level b, x, s, then the coarsest solve's vector, factors and the levels'
// tables -- and forms the V-cycle's matrix.
void setup_dense(PoissonPlan* P, const int* swaps, const double* factors, SpareMatrix* spare) {
  const int nl = static_cast<int>(P->levels.size());
  constexpr size_t tsz = sizeof(double);
  constexpr size_t kSmemLimit = 200 * 1024;
  for(int first = 0; first < nl; ++first) {
    if(P->levels[first].L.count() > kDenseCells || nl - first > kTailMaxLevels) continue;
    TailArgs t{};
    t.count = nl - first;
    size_t cursor = 0;  // elements of T
    const size_t align = 16 / tsz;
    for(int l = first; l < nl; ++l) {
      const Level& lv = P->levels[l];
      TailLevel& tl = t.lv[l - first];
      tl.op = lv.op;
      cursor = (cursor + align - 1) / align * align;
      tl.off = static_cast<int>(cursor);
      cursor += 3 * static_cast<size_t>(lv.L.count());
    }
    cursor = (cursor + align - 1) / align * align;
    t.coarse_off = static_cast<int>(cursor);
    t.coarse_n = P->coarse_n;
    cursor += static_cast<size_t>(P->coarse_n) * sizeof(double) / tsz;
    // staged factors (n^2 doubles) and swaps (n ints) of a coarse solve of
    // at most 32 unknowns
    cursor = (cursor + align - 1) / align * align;
    t.fact_off = static_cast<int>(cursor);
    if(P->coarse_n <= 32)
      cursor += (static_cast<size_t>(P->coarse_n) * P->coarse_n * sizeof(double) +
                 static_cast<size_t>(P->coarse_n) * sizeof(int) + tsz - 1) / tsz;
    // the staged tables of every level but the coarsest
    const size_t tab_off = align16(cursor * tsz);
    std::vector<unsigned char> blob;
    for(int l = first; l + 1 < nl; ++l) {
      const Level& lv = P->levels[l];
      const Level& cv = P->levels[l + 1];
      TailLevel& tl = t.lv[l - first];
      const int n = lv.L.count(), nc = cv.L.count();
      tl.nch = lv.rx * lv.ry * lv.rz;
      tl.tab = static_cast<int>(blob.size());
      const TailTabLayout lay = tail_tab_layout(n, nc, tl.nch, tsz);
      blob.resize(blob.size() + lay.bytes, 0);
      unsigned char* base = blob.data() + tl.tab;
      int16_t* nbr = reinterpret_cast<int16_t*>(base + lay.nbr);
      int16_t* parent = reinterpret_cast<int16_t*>(base + lay.parent);
      int16_t* child = reinterpret_cast<int16_t*>(base + lay.child);
      const std::vector<double> tinv = inverse_diagonal_table(lv.g, P->pbc);
      // nb_lo / nb_hi on the host: neighbour, periodic image or the cell itself,
      // with -1 for a homogeneous-Dirichlet image
      auto rule = [&](int a, int c, bool hi, int& cc) {
        const int N = lv.L.n(a);
        const bool per = lv.op.periodic[a] != 0;
        const bool dir = (hi ? lv.op.dir_hi[a] : lv.op.dir_lo[a]) != 0;
        const bool in = hi ? c < N - 1 : c > 0;
        cc = in ? (hi ? c + 1 : c - 1) : (per ? (hi ? 0 : N - 1) : c);
        return (in || per || !dir) ? 1 : -1;
      };
      auto cls = [](int c, int N) { return N == 1 ? 3 : (c == 0 ? 1 : (c == N - 1 ? 2 : 0)); };
      for(int k = 0; k < lv.L.nz; ++k)
        for(int j = 0; j < lv.L.ny; ++j)
          for(int i = 0; i < lv.L.nx; ++i) {
            const int q = lv.L.idx(i, j, k);
            int cc;
            int sg = rule(0, i, false, cc);
            nbr[q] = static_cast<int16_t>(sg * (lv.L.idx(cc, j, k) + 1));
            sg = rule(0, i, true, cc);
            nbr[n + q] = static_cast<int16_t>(sg * (lv.L.idx(cc, j, k) + 1));
            sg = rule(1, j, false, cc);
            nbr[2 * n + q] = static_cast<int16_t>(sg * (lv.L.idx(i, cc, k) + 1));
            sg = rule(1, j, true, cc);
            nbr[3 * n + q] = static_cast<int16_t>(sg * (lv.L.idx(i, cc, k) + 1));
            sg = rule(2, k, false, cc);
            nbr[4 * n + q] = static_cast<int16_t>(sg * (lv.L.idx(i, j, cc) + 1));
            sg = rule(2, k, true, cc);
            nbr[5 * n + q] = static_cast<int16_t>(sg * (lv.L.idx(i, j, cc) + 1));
            parent[q] = static_cast<int16_t>(cv.L.idx(i / lv.rx, j / lv.ry, k / lv.rz));
            base[lay.cls + q] =
                static_cast<unsigned char>(cls(i, lv.L.nx) + 4 * cls(j, lv.L.ny) + 16 * cls(k, lv.L.nz));
          }
      for(int c = 0; c < 64; ++c) reinterpret_cast<double*>(base + lay.itab)[c] = tinv[c];
      for(int K = 0; K < cv.L.nz; ++K)
        for(int J = 0; J < cv.L.ny; ++J)
          for(int I = 0; I < cv.L.nx; ++I) {
            int c = 0;
            const int Q = cv.L.idx(I, J, K);
            for(int dz = 0; dz < lv.rz; ++dz)
              for(int dy = 0; dy < lv.ry; ++dy)
                for(int dx = 0; dx < lv.rx; ++dx)
                  child[Q * tl.nch + c++] =
                      static_cast<int16_t>(lv.L.idx(I * lv.rx + dx, J * lv.ry + dy, K * lv.rz + dz));
          }
    }
    t.tab_off = static_cast<int>(tab_off);
    t.tab_bytes = static_cast<int>(blob.size());
    const size_t bytes = tab_off + blob.size();
    if(bytes > kSmemLimit) continue;
    DeviceBytes tabs(blob.size());
    if(!blob.empty())
      OFB_CHECK(cudaMemcpy(tabs.p, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    t.tabs = static_cast<const unsigned char*>(tabs.p);
    t.swaps = swaps;
    t.factors = factors;
    t.zm = P->zero_mean;
    const int n = P->levels[first].L.count();
    auto columns = [&](auto* G, auto kern) {
      // the limit itself, whatever this plan needs: the attribute is the kernel's
      OFB_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit)));
      kern<<<n, kTailThreads, bytes>>>(t, G);
      OFB_LAUNCH_CHECK("k_dense_columns");
    };
    const size_t gbytes = static_cast<size_t>(n) * n * (P->precision == 1 ? sizeof(float) : sizeof(double));
    if(spare != nullptr && spare->bytes == gbytes) std::swap(P->dense, spare->p);
    else OFB_CHECK(cudaMalloc(&P->dense, gbytes));
    P->dense_bytes = gbytes;
    P->bytes += gbytes;
    if(P->precision == 1) columns(static_cast<float*>(P->dense), k_dense_columns<float>);
    else columns(static_cast<double*>(P->dense), k_dense_columns<double>);
    OFB_CHECK(cudaStreamSynchronize(nullptr));  // the tables and factors are freed on return
    P->tail_first = first;
    return;
  }
  throw std::invalid_argument("the coarsest multigrid level does not fit the dense solve");
}

// The instantiation for the plan's boundary conditions: sign images where a
// face is Dirichlet, one diagonal value where every face is periodic.
template <typename T>
auto descend_kernel(const PoissonPlan* P, bool flat) {
  using namespace march;
  if(!P->zero_mean) return flat ? k_descend<T, true, false, true> : k_descend<T, true, false, false>;
  if(P->all_periodic) return flat ? k_descend<T, false, true, true> : k_descend<T, false, true, false>;
  return flat ? k_descend<T, false, false, true> : k_descend<T, false, false, false>;
}

template <typename T, bool FINE, bool PAIRS>
auto ascend_kernel_of(const PoissonPlan* P, bool flat) {
  using namespace march;
  if(!P->zero_mean)
    return flat ? k_ascend<T, true, false, true, FINE, PAIRS> : k_ascend<T, true, false, false, FINE, PAIRS>;
  if(P->all_periodic)
    return flat ? k_ascend<T, false, true, true, FINE, PAIRS> : k_ascend<T, false, true, false, FINE, PAIRS>;
  return flat ? k_ascend<T, false, false, true, FINE, PAIRS> : k_ascend<T, false, false, false, FINE, PAIRS>;
}

template <typename T>
auto ascend_kernel(const PoissonPlan* P, bool flat, bool fine, bool pairs) {
  if(fine) return pairs ? ascend_kernel_of<T, true, true>(P, flat) : ascend_kernel_of<T, true, false>(P, flat);
  return pairs ? ascend_kernel_of<T, false, true>(P, flat) : ascend_kernel_of<T, false, false>(P, flat);
}

template <typename T>
auto direction_kernel(const PoissonPlan* P, bool flat) {
  using namespace march;
  if(!P->zero_mean) return flat ? k_direction<T, true, true> : k_direction<T, true, false>;
  return flat ? k_direction<T, false, true> : k_direction<T, false, false>;
}

template <typename T>
auto advance_kernel(const PoissonPlan* P, bool flat) {
  using namespace march;
  if(!P->zero_mean) return flat ? k_advance<T, true, true> : k_advance<T, true, false>;
  return flat ? k_advance<T, false, true> : k_advance<T, false, false>;
}

template <bool START>
auto residual_kernel(const PoissonPlan* P, bool flat) {
  using namespace march;
  if(!P->zero_mean) return flat ? k_residual<true, true, START> : k_residual<true, false, START>;
  return flat ? k_residual<false, true, START> : k_residual<false, false, START>;
}

constexpr int kMarchSmem = 224 * 1024;

// Lets every instantiation use the largest tile's shared memory.
template <typename T>
void march_attributes(const PoissonPlan* P) {
  auto attr = [](auto kern) {
    OFB_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMarchSmem));
  };
  for(const bool flat : {false, true}) {
    attr(descend_kernel<T>(P, flat));
    attr(direction_kernel<T>(P, flat));
    attr(advance_kernel<T>(P, flat));
    attr(residual_kernel<true>(P, flat));
    attr(residual_kernel<false>(P, flat));
    for(const bool fine : {false, true})
      for(const bool pairs : {false, true}) attr(ascend_kernel<T>(P, flat, fine, pairs));
  }
}

// Tile and grid of a march kernel on one level: the split with the least
// modelled time.  A block of `threads` marches chunk + 3 planes (its halo
// planes and the pipeline's fill included); an SM takes about kPlaneLatency
// cycles for a plane when few threads are resident (barrier, shared-memory and
// arithmetic latency) and kThreadCycles per resident thread when many are
// (measured: 510 threads, 1000 cycles per plane at 256^3), and the blocks run
// in waves of what the SMs hold at once.  Small levels so get many thin
// chunks, large ones tiles near 64 x 26 with long chunks.
constexpr double kPlaneLatency = 500.0, kThreadCycles = 2.0;
// Resident threads of the kernels on grids one cell deep (56-80 registers).
constexpr int kFlatResident = 768;

template <typename T>
void plan_tile(const CLay& L, int halo_rows, int rz, int streams, int fields, int sms, march::Tile& best,
               dim3& grid) {
  constexpr int W = march::kW<T>;
  auto even = [](int v) { return (v + 1) / 2 * 2; };
  const bool flat = L.nz == 1;
  double best_cost = 0.0;
  bool found = false;
  int last_ix = 0;
  for(int ntx = 1; ntx <= (L.nx + 7) / 8 || ntx == 1; ++ntx) {
    march::Tile t{};
    t.ix = ((L.nx + ntx - 1) / ntx + W - 1) / W * W;
    if(t.ix == last_ix) continue;
    last_ix = t.ix;
    t.px = t.ix / W + 2;
    if(t.px > march::kPX) continue;
    t.tx = (L.nx + t.ix - 1) / t.ix;
    // the most rows that a block's threads and its shared memory take (narrow
    // grids: a row's shared memory has a fixed length)
    auto smem_of = [&](int rows) {
      t.ey = rows + 2 * halo_rows;
      return march::smem_bytes<T>(t, streams, fields, flat, fields == 2);
    };
    int max_rows = march::kMaxThreads / t.px * 2 - 2 * halo_rows;
    while(max_rows > 2 && smem_of(max_rows) > kMarchSmem) max_rows -= 2;
    if(max_rows < 2) continue;
    int last_iy = 0;
    const int nty0 = (L.ny + max_rows - 1) / max_rows;
    for(int nty = nty0; nty <= std::max(nty0, (L.ny + 3) / 4) && nty < nty0 + 64; ++nty) {
      t.iy = std::min(even((L.ny + nty - 1) / nty), max_rows);
      if(t.iy == last_iy) continue;
      last_iy = t.iy;
      const size_t smem = smem_of(t.iy);
      if(smem > kMarchSmem) continue;
      const int threads = t.px * t.ey / 2;
      const int resident = std::min<int>({(flat ? kFlatResident : march::kMaxThreads) / ((threads + 31) / 32 * 32),
                                          static_cast<int>(228 * 1024 / (smem + 2048)), 16});
      if(resident < 1) continue;
      const long long tiles = static_cast<long long>(t.tx) * ((L.ny + t.iy - 1) / t.iy);
      if(tiles > kMaxBlocks) continue;
      const int units = (L.nz + rz - 1) / rz;
      for(int nch = 1; nch <= units && tiles * nch <= kMaxBlocks; nch < 48 ? ++nch : nch *= 2) {
        t.chunk = (units + nch - 1) / nch * rz;
        const long long blocks = tiles * ((L.nz + t.chunk - 1) / t.chunk);
        const long long waves = (blocks + static_cast<long long>(sms) * resident - 1) / (static_cast<long long>(sms) * resident);
        const long long per_sm = std::min<long long>(resident, (blocks + sms - 1) / sms);
        const double plane = std::max(kPlaneLatency, kThreadCycles * static_cast<double>(per_sm) * threads);
        const double cost = static_cast<double>(waves) * (flat ? 3 : t.chunk + 3) * plane;
        if(!found || cost < best_cost) {
          found = true;
          best_cost = cost;
          best = t;
          grid = dim3(static_cast<unsigned>(tiles), static_cast<unsigned>((L.nz + t.chunk - 1) / t.chunk), 1);
        }
        if(flat) break;
      }
    }
  }
  if(!found) throw std::invalid_argument("grid too large for the pressure solve's tiles");
}

}  // namespace

PoissonPlan* poisson_plan_create(const Grid& g, const PBC& pbc_in, int precision, SpareMatrix* spare) {
  struct FreeSpare {
    SpareMatrix* m;
    ~FreeSpare() {
      if(m != nullptr) cudaFree(m->p);
    }
  } free_spare{spare};
  // destroyed with the function's scope unless it gets to its end
  std::unique_ptr<PoissonPlan, void (*)(PoissonPlan*)> plan(new PoissonPlan(), poisson_plan_destroy);
  PoissonPlan* const P = plan.get();
  P->g = g;
  // homogeneous_boundary_conditions (linsolve/poisson_solver.cpp:164-173)
  P->pbc = pbc_in;
  for(int f = 0; f < 6; ++f) {
    P->pbc.value[f] = 0.0;
    P->pbc.gradient[f] = 0.0;
  }
  P->precision = precision;
  P->zero_mean = 1;
  for(int f = 0; f < 6; ++f)
    if(pbc_in.type[f] == kPDirichlet) P->zero_mean = 0;
  const size_t tsz = precision == 1 ? sizeof(float) : sizeof(double);

  // build_hierarchy (linsolve/poisson_solver.cpp:316-384)
  Grid cur = g;
  for(;;) {
    Level lv;
    lv.g = cur;
    lv.L = make_clay(cur.nx, cur.ny, cur.nz);
    lv.op = make_op(cur, P->pbc);
    P->levels.push_back(lv);
    if(!(can_coarsen_axis(cur.nx) || can_coarsen_axis(cur.ny) || can_coarsen_axis(cur.nz))) break;
    Grid c = cur;
    if(can_coarsen_axis(cur.nx)) { c.nx = cur.nx / 2; c.dx = 2.0 * cur.dx; }
    if(can_coarsen_axis(cur.ny)) { c.ny = cur.ny / 2; c.dy = 2.0 * cur.dy; }
    if(can_coarsen_axis(cur.nz)) { c.nz = cur.nz / 2; c.dz = 2.0 * cur.dz; }
    if(c.nx == cur.nx && c.ny == cur.ny && c.nz == cur.nz) break;
    Level& prev = P->levels.back();
    prev.rx = cur.nx == c.nx ? 1 : 2;
    prev.ry = cur.ny == c.ny ? 1 : 2;
    prev.rz = cur.nz == c.nz ? 1 : 2;
    cur = c;
  }
  const int nl = static_cast<int>(P->levels.size());
  for(int l = 0; l < nl; ++l) {
    Level& lv = P->levels[l];
    const size_t n = lv.L.count();
    OFB_CHECK(cudaMalloc(&lv.a, n * tsz));
    OFB_CHECK(cudaMalloc(&lv.x, n * tsz));
    P->bytes += 2 * n * tsz;
    if(l > 0) {
      OFB_CHECK(cudaMalloc(&lv.b, n * tsz));
      P->bytes += n * tsz;
    }
    std::vector<double> t = inverse_diagonal_table(lv.g, P->pbc);
    OFB_CHECK(cudaMalloc(&lv.invd, 64 * sizeof(double)));
    OFB_CHECK(cudaMemcpy(lv.invd, t.data(), 64 * sizeof(double), cudaMemcpyHostToDevice));
    lv.op.invd = lv.invd;
  }
  OFB_CHECK(cudaMalloc(&P->ls, nl * sizeof(LevelScalars)));
  OFB_CHECK(cudaMemset(P->ls, 0, nl * sizeof(LevelScalars)));

  // coarsest-grid elimination (direct_coarse_solve / gaussian_elimination,
  // linsolve/poisson_solver.cpp:482-567), done once on the host
  const Level& co = P->levels.back();
  const int n = co.L.count();
  if(n > kMaxCoarse) {
    throw std::invalid_argument("coarsest multigrid level has " + std::to_string(n) +
                                " unknowns; at most " + std::to_string(kMaxCoarse) +
                                " are supported");
  }
  P->coarse_n = n;
  std::vector<double> m(static_cast<size_t>(n) * n, 0.0), e(n, 0.0), img(n, 0.0);
  for(int col = 0; col < n; ++col) {
    std::fill(e.begin(), e.end(), 0.0);
    e[col] = 1.0;
    host_apply(co.g, P->pbc, e, img);
    for(int row = 0; row < n; ++row) m[static_cast<size_t>(row) * n + col] = img[row];
  }
  if(P->zero_mean)
    for(int col = 0; col < n; ++col) m[static_cast<size_t>(n - 1) * n + col] = 1.0;
  std::vector<int> swaps(n);
  for(int piv = 0; piv < n; ++piv) {
    int best = piv;
    double best_abs = std::fabs(m[static_cast<size_t>(piv) * n + piv]);
    for(int row = piv + 1; row < n; ++row) {
      const double cand = std::fabs(m[static_cast<size_t>(row) * n + piv]);
      if(cand > best_abs) {
        best = row;
        best_abs = cand;
      }
    }
    if(best_abs < kSmallNumber) {
      throw std::runtime_error("direct coarse solve encountered a singular matrix");
    }
    swaps[piv] = best;
    // Columns left of the pivot hold the multipliers of earlier steps; they
    // stay with their row position so the device replays the eliminations
    // on the right-hand side in the reference's order.
    if(best != piv)
      for(int c = piv; c < n; ++c)
        std::swap(m[static_cast<size_t>(piv) * n + c], m[static_cast<size_t>(best) * n + c]);
    const double inv = 1.0 / m[static_cast<size_t>(piv) * n + piv];
    for(int row = piv + 1; row < n; ++row) {
      const double factor = m[static_cast<size_t>(row) * n + piv] * inv;
      if(std::fabs(factor) < kSmallNumber) {
        m[static_cast<size_t>(row) * n + piv] = 0.0;
        continue;
      }
      for(int c = piv + 1; c < n; ++c)
        m[static_cast<size_t>(row) * n + c] -= factor * m[static_cast<size_t>(piv) * n + c];
      m[static_cast<size_t>(row) * n + piv] = factor;  // keep the multiplier
    }
  }
  {
    DeviceBytes dswaps(n * sizeof(int)), dfact(static_cast<size_t>(n) * n * sizeof(double));
    OFB_CHECK(cudaMemcpy(dswaps.p, swaps.data(), n * sizeof(int), cudaMemcpyHostToDevice));
    OFB_CHECK(cudaMemcpy(dfact.p, m.data(), static_cast<size_t>(n) * n * sizeof(double), cudaMemcpyHostToDevice));
    setup_dense(P, static_cast<const int*>(dswaps.p), static_cast<const double*>(dfact.p), spare);
  }

  const size_t nf = P->levels[0].L.count();
  OFB_CHECK(cudaMalloc(&P->b, nf * sizeof(double)));
  OFB_CHECK(cudaMalloc(&P->x, nf * sizeof(double)));
  OFB_CHECK(cudaMalloc(&P->r, nf * sizeof(double)));
  OFB_CHECK(cudaMalloc(&P->p, nf * sizeof(double)));
  OFB_CHECK(cudaMemset(P->p, 0, nf * sizeof(double)));
  OFB_CHECK(cudaMalloc(&P->p2, nf * sizeof(double)));
  OFB_CHECK(cudaMemset(P->p2, 0, nf * sizeof(double)));
  P->bytes += 5 * nf * sizeof(double);
  if(precision == 1) {
    for(float** v : {&P->r32, &P->e32, &P->p32, &P->p32b}) {
      OFB_CHECK(cudaMalloc(v, nf * sizeof(float)));
      OFB_CHECK(cudaMemset(*v, 0, nf * sizeof(float)));
    }
    OFB_CHECK(cudaMalloc(&P->sc_in, sizeof(SolveScalars)));
    OFB_CHECK(cudaMemset(P->sc_in, 0, sizeof(SolveScalars)));
    P->bytes += 4 * nf * sizeof(float);
  }
  {
    int dev = 0;
    OFB_CHECK(cudaGetDevice(&dev));
    OFB_CHECK(cudaDeviceGetAttribute(&P->sms, cudaDevAttrMultiProcessorCount, dev));
  }
  P->all_periodic = true;
  for(int f = 0; f < 6; ++f)
    if(P->pbc.type[f] != kPPeriodic) P->all_periodic = false;
  for(int l = 0; l < P->tail_first; ++l)
    (precision == 1 ? plan_tile<float> : plan_tile<double>)(P->levels[l].L, 2, P->levels[l].rz, 2, 2, P->sms,
                                                            P->levels[l].tile, P->levels[l].tgrid);
  (precision == 1 ? plan_tile<float> : plan_tile<double>)(P->levels[0].L, 1, 1, 3, 1, P->sms, P->cg_tile, P->cg_grid);
  plan_tile<double>(P->levels[0].L, 1, 1, 2, 1, P->sms, P->res_tile, P->res_grid);
  if(precision == 1) march_attributes<float>(P);
  else march_attributes<double>(P);
  const char* no_graph = std::getenv("ORCHARD_B200_NO_GRAPH");
  P->use_graph = !(no_graph != nullptr && no_graph[0] == '1');
  // what was set up above went through the default stream, with which the
  // context's stream does not synchronise: behind another thread's plan it
  // would still be on its way when the first solve runs
  OFB_CHECK(cudaStreamSynchronize(nullptr));
  return plan.release();
}

void poisson_plan_destroy(PoissonPlan* P) {
  if(P == nullptr) return;
  for(Level& lv : P->levels) {
    cudaFree(lv.a);
    cudaFree(lv.x);
    cudaFree(lv.b);
    cudaFree(lv.invd);
  }
  if(P->exec) cudaGraphExecDestroy(P->exec);
  if(P->graph) cudaGraphDestroy(P->graph);
  cudaFree(P->hist);
  cudaFree(P->ls);
  cudaFree(P->b);
  cudaFree(P->x);
  cudaFree(P->r);
  cudaFree(P->p);
  cudaFree(P->r32);
  cudaFree(P->e32);
  cudaFree(P->p32);
  cudaFree(P->p2);
  cudaFree(P->p32b);
  cudaFree(P->sc_in);
  cudaFree(P->dense);
  delete P;
}

SpareMatrix poisson_release_matrix(PoissonPlan* P) {
  SpareMatrix m;
  if(P != nullptr) {
    std::swap(m.p, P->dense);
    m.bytes = P->dense_bytes;
  }
  return m;
}

int poisson_levels(const PoissonPlan* P) { return static_cast<int>(P->levels.size()); }
int poisson_coarse_unknowns(const PoissonPlan* P) { return P->coarse_n; }
size_t poisson_device_bytes(const PoissonPlan* P) { return P->bytes; }
double* poisson_b(PoissonPlan* P) { return P->b; }
double* poisson_x(PoissonPlan* P) { return P->x; }

namespace {

// v_cycle (linsolve/poisson_solver.cpp:597-633) from level l; the finest
// level's rhs is the CG residual r0 (type V, shift sc->sr).
template <typename T, typename V>
void v_cycle(PoissonPlan* P, int l, const V* r0, SolveScalars* sc, RedBuf rb, cudaStream_t s) {
  Level& lv = P->levels[l];
  LevelScalars* ls = P->ls + l;
  const double* sb_ptr = l == 0 ? &sc->sr : &ls->sb;  // ls->sb stays 0 (k_descend)
  T* a = static_cast<T*>(lv.a);
  T* x = static_cast<T*>(lv.x);
  if(l == P->tail_first) {
    ProfScope ps(l == 0 ? kKCoarseSolve : kKCoarseLevels, s);
    const int n = lv.L.count();
    const dim3 grid((n + kDenseRows - 1) / kDenseRows);
    const T* G = static_cast<const T*>(P->dense);
    if(l == 0)
      launch_pdl(k_dense_apply<T, V>, grid, kDenseThreads, 0, s, n, G, r0, x, ls, sc, rb);
    else
      launch_pdl(k_dense_apply<T, T>, grid, kDenseThreads, 0, s, n, G, static_cast<const T*>(lv.b), x, ls,
                 static_cast<SolveScalars*>(nullptr), rb);
    OFB_LAUNCH_CHECK("k_dense_apply");
    return;
  }
  Level& cv = P->levels[l + 1];
  const T* b = l == 0 ? static_cast<const T*>(r0) : static_cast<const T*>(lv.b);
  const size_t smem1 = march::smem_bytes<T>(lv.tile, 1, 2, lv.L.nz == 1),
               smem2 = march::smem_bytes<T>(lv.tile, 2, 2, lv.L.nz == 1, true);
  const int threads = lv.tile.px * lv.tile.ey / 2;
  {
    ProfScope ps(l == 0 ? kKSmoothFirstFine : kKCoarseLevels, s);
    launch_pdl(descend_kernel<T>(P, lv.L.nz == 1), lv.tgrid, threads, smem1, s, lv.op, cv.L, lv.tile, b, sb_ptr,
               a, static_cast<T*>(cv.b), lv.rx, lv.ry, lv.rz);
  }
  if(l == 0) {
    // the coarse levels are short dependent launches: time them as one chain
    // (one event pair per V-cycle) so that the measurement does not add an
    // event pair's overhead to each of them
    ProfSpan span(kKCoarseLevels, s);
    v_cycle<T, V>(P, l + 1, r0, sc, rb, s);
  } else {
    v_cycle<T, V>(P, l + 1, r0, sc, rb, s);
  }
  {
    ProfScope ps(l == 0 ? kKSmoothFine : kKCoarseLevels, s);
    launch_pdl(ascend_kernel<T>(P, lv.L.nz == 1, l == 0, lv.rx == 2 && lv.ry == 2), lv.tgrid, threads, smem2, s, lv.op, cv.L, lv.tile, b,
               sb_ptr, static_cast<const T*>(a), static_cast<const T*>(cv.x), x, lv.rx - 1, lv.ry - 1,
               lv.rz - 1, ls, sc, rb);
  }
  OFB_LAUNCH_CHECK("v_cycle");
}

// The vectors of one CG loop: FP64 for the reference's solve, FP32 for the
// inner solves of the mixed path's defect correction.
template <typename V>
struct CGVec {
  V *x, *r, *p, *p2;  // p and p2 alternate (march::Direction)
};

CGVec<double> cg64(PoissonPlan* P) { return CGVec<double>{P->x, P->r, P->p, P->p2}; }

// Initial residual and convergence test (linsolve/poisson_solver.cpp:717-739).
void enqueue_start(PoissonPlan* P, const march::SolveStart& start, SolveScalars* sc, RedBuf rb, cudaStream_t s,
                   bool zero_guess) {
  const Level& l0 = P->levels[0];
  ProfScope ps(kKInitResidual, s);
  if(zero_guess) {
    const int n = l0.L.count();
    const int blocks = std::min(kTargetBlocks, (n + kFlatThreads - 1) / kFlatThreads);
    k_start_from_zero<<<blocks, kFlatThreads, 0, s>>>(n, P->b, P->x, P->r, sc, start, rb);
    OFB_LAUNCH_CHECK("k_start_from_zero");
    return;
  }
  const march::Tile& t = P->res_tile;
  launch_pdl(residual_kernel<true>(P, l0.L.nz == 1), P->res_grid, t.px * t.ey / 2, march::smem_bytes<double>(t, 2, 1, l0.L.nz == 1),
             s, l0.op, t, P->x, P->b, P->r, sc, static_cast<const SolveScalars*>(nullptr), start, rb);
  OFB_LAUNCH_CHECK("k_residual");
}

// One body of the rotated PCG loop: z = M r, p = z + beta p and p.Ap, x/r update
// and the convergence test -- the reference's iteration (:750-806) with the
// preconditioner moved to the top; the body count is the reference's
// iteration count, and the first body forms p = z as the reference does
// before its loop (:741-749).
template <typename T, typename V>
void enqueue_body(PoissonPlan* P, const CGVec<V>& v, SolveScalars* sc, RedBuf rb, cudaStream_t s,
                  cudaGraphConditionalHandle cond) {
  const Level& l0 = P->levels[0];
  v_cycle<T, V>(P, 0, v.r, sc, rb, s);
  const march::Tile& t = P->cg_tile;
  const int threads = t.px * t.ey / 2;
  const bool flat = l0.L.nz == 1;
  const march::Direction<V> d{{v.p, v.p2}};
  {
    ProfScope ps(kKApplyAp, s);
    launch_pdl(direction_kernel<V>(P, flat), P->cg_grid, threads, march::smem_bytes<V>(t, 2, 1, flat), s, l0.op, t,
               static_cast<const V*>(l0.x), P->ls, d, sc, rb);
  }
  {
    ProfScope ps(kKUpdateXr, s);
    launch_pdl(advance_kernel<V>(P, flat), P->cg_grid, threads, march::smem_bytes<V>(t, 3, 1, flat), s, l0.op, t, d,
               v.x, v.r, sc, rb, cond);
  }
  OFB_LAUNCH_CHECK("pcg body");
}

// A stream's capture with the launches counted into `counts`; an exception on
// the way ends both, so the stream and the profiler stay usable.
class Capture {
 public:
  Capture(cudaStream_t s, long long* counts, cudaGraph_t into) : s_(s) {
    if(into != nullptr)
      OFB_CHECK(cudaStreamBeginCaptureToGraph(s, into, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    else
      OFB_CHECK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    open_ = true;
    owns_ = into == nullptr;
    prof_capture_begin(counts);
  }
  Capture(const Capture&) = delete;
  Capture& operator=(const Capture&) = delete;
  cudaGraph_t end() {
    cudaGraph_t g = nullptr;
    open_ = false;
    prof_capture_end();
    OFB_CHECK(cudaStreamEndCapture(s_, &g));
    return g;
  }
  ~Capture() {
    if(!open_) return;
    cudaGraph_t g = nullptr;
    prof_capture_end();
    cudaStreamEndCapture(s_, &g);
    if(owns_ && g != nullptr) cudaGraphDestroy(g);
    cudaGetLastError();
  }

 private:
  cudaStream_t s_;
  bool open_ = false, owns_ = false;
};

// A loop as one graph: pre -> WHILE(cont) { body }.  pre and body are
// enqueue callbacks taking the conditional handle; the loop is bounded by the
// iteration limit the body enforces (it clears the condition), so the graph
// always terminates.
template <typename Pre, typename Body>
cudaGraphExec_t build_loop_graph(PoissonPlan* P, cudaStream_t s, Pre pre, Body body,
                                 cudaGraph_t* graph_out) {
  struct Graph {
    cudaGraph_t g = nullptr;
    ~Graph() {
      if(g != nullptr) cudaGraphDestroy(g);
    }
  } graph;
  OFB_CHECK(cudaGraphCreate(&graph.g, 0));
  const cudaGraph_t g = graph.g;
  cudaGraphConditionalHandle cond = 0;
  OFB_CHECK(cudaGraphConditionalHandleCreate(&cond, g, 0, cudaGraphCondAssignDefault));
  for(int i = 0; i < kKernelCount; ++i) P->pre_counts[i] = P->body_counts[i] = 0;
  std::vector<cudaGraphNode_t> leaf;
  {
    Capture c(s, P->pre_counts, g);
    pre(cond);
    cudaStreamCaptureStatus status;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    OFB_CHECK(cudaStreamGetCaptureInfo(s, &status, nullptr, nullptr, &deps, &ndeps));
    leaf.assign(deps, deps + ndeps);
    c.end();
  }
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = cond;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t wnode;
  OFB_CHECK(cudaGraphAddNode(&wnode, g, leaf.data(), leaf.size(), &cp));
  {
    Capture c(s, P->body_counts, cp.conditional.phGraph_out[0]);
    body(cond);
    c.end();
  }
  cudaGraphExec_t exec = nullptr;
  OFB_CHECK(cudaGraphInstantiate(&exec, g, 0));
  *graph_out = g;
  graph.g = nullptr;
  return exec;
}

void ensure_history(PoissonPlan* P, int max_iterations) {
  if(P->hist_cap < max_iterations + 1) {
    if(P->hist) cudaFree(P->hist);
    P->hist = nullptr;
    OFB_CHECK(cudaMalloc(&P->hist, sizeof(double) * (max_iterations + 1)));
    P->hist_cap = max_iterations + 1;
  }
}

march::SolveStart solve_start(PoissonPlan* P, int max_iterations, double tolerance) {
  ensure_history(P, max_iterations);
  return march::SolveStart{tolerance, max_iterations, P->levels[0].L.count(), P->zero_mean, P->hist, P->hist_cap};
}

bool loop_on_device(const PoissonPlan* P) { return P->use_graph && !prof_enabled(); }

// Enqueues an FP64 solve as one graph launch after its start.
template <typename T>
void enqueue_solve(PoissonPlan* P, int max_iterations, double tolerance, SolveScalars* sc, RedBuf rb,
                   cudaStream_t s, bool zero_guess) {
  enqueue_start(P, solve_start(P, max_iterations, tolerance), sc, rb, s, zero_guess);
  if(P->exec == nullptr) {
    const CGVec<double> v = cg64(P);
    P->exec = build_loop_graph(
        P, s,
        [&](cudaGraphConditionalHandle c) {
          k_loop_gate<<<1, 1, 0, s>>>(sc, c);
          OFB_LAUNCH_CHECK("k_loop_gate");
        },
        [&](cudaGraphConditionalHandle c) { enqueue_body<T, double>(P, v, sc, rb, s, c); }, &P->graph);
  }
  OFB_CHECK(cudaGraphLaunch(P->exec, s));
}

template <typename T>
void solve_impl(PoissonPlan* P, int max_iterations, double tolerance, SolveScalars* sc,
                SolveScalars* host, RedBuf rb, cudaStream_t s, double* history, int history_cap, bool zero_guess) {
  auto read = [&] {
    OFB_CHECK(cudaMemcpyAsync(host, sc, sizeof(SolveScalars), cudaMemcpyDeviceToHost, s));
    OFB_CHECK(cudaStreamSynchronize(s));
    prof_collect();
  };
  if(loop_on_device(P)) {
    enqueue_solve<T>(P, max_iterations, tolerance, sc, rb, s, zero_guess);
    read();
    poisson_account(P, *host);
  } else {
    const CGVec<double> v = cg64(P);
    enqueue_start(P, solve_start(P, max_iterations, tolerance), sc, rb, s, zero_guess);
    for(read(); host->cont; read()) enqueue_body<T, double>(P, v, sc, rb, s, 0);
  }
  if(history != nullptr && history_cap > 0) {
    const int n = std::min(history_cap, std::min(host->iterations + 1, P->hist_cap));
    OFB_CHECK(cudaMemcpy(history, P->hist, sizeof(double) * n, cudaMemcpyDeviceToHost));
  }
}

// ---------------------------------------------------------------------------
// Mixed path: defect correction.  The outer loop is FP64 -- residual
// r = b - A x, its norm and the convergence test against the reference's
// relative tolerance, the update x += e, the mean shifts -- and each inner
// solve A e = r runs the same MG-PCG entirely in FP32 storage and arithmetic
// (V-cycle and CG vectors; dot products and means accumulated in FP64) on the
// residual scaled to unit RMS, to a relative residual of kInnerTol.  The
// reported iteration count is the total number of inner iterations.
// ---------------------------------------------------------------------------
constexpr double kInnerTol = 1.0e-4;
constexpr int kInnerMaxIt = 60;

template <typename T>
void solve_dc(PoissonPlan* P, int max_iterations, double tolerance, SolveScalars* sc,
              SolveScalars* host, RedBuf rb, cudaStream_t s, double* history, int history_cap, bool zero_guess) {
  const Level& l0 = P->levels[0];
  const Launch3 ln = launch3(l0.L.nx, l0.L.ny, l0.L.nz, kReducingBlocks);
  const march::SolveStart start = solve_start(P, max_iterations, tolerance);
  enqueue_start(P, start, sc, rb, s, zero_guess);
  OFB_CHECK(cudaMemcpyAsync(host, sc, sizeof(SolveScalars), cudaMemcpyDeviceToHost, s));
  OFB_CHECK(cudaStreamSynchronize(s));
  const CGVec<float> v{P->e32, P->r32, P->p32, P->p32b};
  SolveScalars* si = P->sc_in;
  auto pre = [&](cudaGraphConditionalHandle c) {
    ProfScope ps(kKDefectCorrection, s);
    k_dc_to_inner<<<ln.grid, ln.block, 0, s>>>(l0.L, P->r, sc, P->r32, P->e32, si, kInnerTol,
                                               kInnerMaxIt, ln.kchunk, rb, c);
    OFB_LAUNCH_CHECK("k_dc_to_inner");
  };
  auto body = [&](cudaGraphConditionalHandle c) { enqueue_body<T, float>(P, v, si, rb, s, c); };
  auto post = [&]() {
    ProfScope ps(kKDefectCorrection, s, 2);
    k_dc_update_x<<<ln.grid, ln.block, 0, s>>>(l0.L, P->x, P->e32, sc, si, ln.kchunk, rb);
    const march::Tile& t = P->res_tile;
    launch_pdl(residual_kernel<false>(P, l0.L.nz == 1), P->res_grid, t.px * t.ey / 2,
               march::smem_bytes<double>(t, 2, 1, l0.L.nz == 1), s, l0.op, t, P->x, P->b, P->r, sc,
               static_cast<const SolveScalars*>(si), start, rb);
    OFB_LAUNCH_CHECK("defect correction update");
  };
  const bool use_graph = loop_on_device(P);
  long long inner_runs = 0;
  while(host->cont) {
    if(use_graph) {
      if(P->exec == nullptr) P->exec = build_loop_graph(P, s, pre, body, &P->graph);
      OFB_CHECK(cudaGraphLaunch(P->exec, s));
      post();
    } else {
      pre(0);
      SolveScalars hi{};
      OFB_CHECK(cudaMemcpyAsync(&hi, si, sizeof(SolveScalars), cudaMemcpyDeviceToHost, s));
      OFB_CHECK(cudaStreamSynchronize(s));
      prof_collect();
      while(hi.cont) {
        body(0);
        OFB_CHECK(cudaMemcpyAsync(&hi, si, sizeof(SolveScalars), cudaMemcpyDeviceToHost, s));
        OFB_CHECK(cudaStreamSynchronize(s));
        prof_collect();
      }
      post();
    }
    OFB_CHECK(cudaMemcpyAsync(host, sc, sizeof(SolveScalars), cudaMemcpyDeviceToHost, s));
    OFB_CHECK(cudaStreamSynchronize(s));
    if(use_graph) {
      prof_add_counts(P->pre_counts, 1);
      prof_add_counts(P->body_counts, host->body_runs - inner_runs);
      inner_runs = host->body_runs;
    }
    prof_collect();
  }
  if(history != nullptr && history_cap > 0) {
    const int n = std::min(history_cap, std::min(host->outer + 1, P->hist_cap));
    OFB_CHECK(cudaMemcpy(history, P->hist, sizeof(double) * n, cudaMemcpyDeviceToHost));
  }
}

}  // namespace

void poisson_account(PoissonPlan* P, const SolveScalars& host) {
  prof_add_counts(P->pre_counts, 1);
  prof_add_counts(P->body_counts, host.body_runs);
}

void poisson_solve(PoissonPlan* P, int max_iterations, double tolerance, SolveScalars* sc_dev,
                   SolveScalars* sc_host, RedBuf rb, cudaStream_t s, double* history,
                   int history_cap, bool zero_guess) {
  if(P->precision == 1)
    solve_dc<float>(P, max_iterations, tolerance, sc_dev, sc_host, rb, s, history, history_cap, zero_guess);
  else
    solve_impl<double>(P, max_iterations, tolerance, sc_dev, sc_host, rb, s, history, history_cap, zero_guess);
}

bool poisson_solve_enqueue(PoissonPlan* P, int max_iterations, double tolerance, SolveScalars* sc_dev,
                           SolveScalars* sc_host, RedBuf rb, cudaStream_t s, bool zero_guess) {
  if(P->precision == 1 || !loop_on_device(P)) {
    poisson_solve(P, max_iterations, tolerance, sc_dev, sc_host, rb, s, nullptr, 0, zero_guess);
    return false;
  }
  enqueue_solve<double>(P, max_iterations, tolerance, sc_dev, rb, s, zero_guess);
  return true;
}

double poisson_time_coarse_chain(PoissonPlan* P, RedBuf rb, cudaStream_t s, int reps, int* launches) {
  *launches = 0;
  // a finest level that is the dense one has no chain below it
  if(P->tail_first < 1 || reps < 1) return 0.0;
  long long counts[kKernelCount] = {};
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  {
    Capture c(s, counts, nullptr);
    // levels >= 1 read only their own level data and LevelScalars
    if(P->precision == 1)
      v_cycle<float, float>(P, 1, nullptr, nullptr, rb, s);
    else
      v_cycle<double, double>(P, 1, nullptr, nullptr, rb, s);
    g = c.end();
  }
  for(int i = 0; i < kKernelCount; ++i) *launches += static_cast<int>(counts[i]);
  OFB_CHECK(cudaGraphInstantiate(&ge, g, 0));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  OFB_CHECK(cudaEventCreate(&e0));
  OFB_CHECK(cudaEventCreate(&e1));
  for(int i = 0; i < 3; ++i) OFB_CHECK(cudaGraphLaunch(ge, s));
  OFB_CHECK(cudaEventRecord(e0, s));
  for(int i = 0; i < reps; ++i) OFB_CHECK(cudaGraphLaunch(ge, s));
  OFB_CHECK(cudaEventRecord(e1, s));
  OFB_CHECK(cudaEventSynchronize(e1));
  float ms = 0.0f;
  OFB_CHECK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaGraphExecDestroy(ge);
  cudaGraphDestroy(g);
  return 1000.0 * ms / reps;
}

void launch_compact_to_pressure(const Grid& g, const double* x, const SolveScalars* sc,
                                double* p_padded, cudaStream_t s) {
  dim3 block(32, 8, 1);
  dim3 grid((g.nx + 31) / 32, (g.ny + 7) / 8, g.nz);
  ProfScope ps(kKOther, s);
  k_compact_to_pressure<<<grid, block, 0, s>>>(g, x, sc, p_padded);
  OFB_LAUNCH_CHECK("k_compact_to_pressure");
}

}  // namespace ofb
