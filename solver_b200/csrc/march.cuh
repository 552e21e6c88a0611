// Fused multigrid and CG kernels that march the k planes of a tile.
//
// A block owns an interior tile of ix x iy cells and a chunk of k planes, plus
// a halo of one patch on either x side and two rows on either y side.  A thread
// owns a patch of two rows of W cells (16 bytes: W = 2 in FP64, 4 in FP32;
// whole footprints of coarse cells, so restriction and prolongation are local
// to it) and walks k with its z neighbours in registers; per plane the block
// publishes the fields whose in-plane neighbours it needs in shared memory,
// passes one barrier (the planes alternate between two buffers) and computes.
// Several sweeps are pipelined in one pass, each a plane behind the one it
// reads: the halo shrinks by one cell per sweep, so intermediate vectors are
// never written to memory.
//
// Cells outside the domain are images: the load maps an index to the cell
// whose value it repeats (periodic wrap, or the mirror cell of a
// homogeneous-Neumann wall) and, for a homogeneous-Dirichlet wall, the sign -1
// (neighbor_value, linsolve/poisson_solver.cpp:195-242).  The operator, the
// Jacobi diagonal and the sweeps commute with these reflections, so a sweep on
// image cells gives the images of the sweep's result and the stencils need no
// boundary cases.
//
// Shared memory holds a row's cells by their position in the patch (all first
// cells, then all second ones, ...): a warp's accesses are then consecutive
// words (no bank conflicts).  Rows
// have a fixed stride and the k loop is unrolled by four with every field's
// planes in a ring of four register slots, so that shared-memory addresses are
// immediates and no plane is ever moved between registers: at one patch per
// thread the loop is bound by its instruction count (rotating registers and
// run-time strides took 359 instructions per patch and plane, 75 of them FP64).
#pragma once

#include "kernels.hpp"

#include <type_traits>

namespace ofb {

struct OpInfo {
  CLay L;
  double inv2[3];  // 1 / h^2
  int periodic[3];
  int dir_lo[3], dir_hi[3];  // homogeneous Dirichlet (else Neumann) at each end
  const double* invd;        // 64-entry inverse-diagonal table
};

__device__ __forceinline__ int axis_class(int c, int n) {
  return n == 1 ? 3 : (c == 0 ? 1 : (c == n - 1 ? 2 : 0));
}

namespace march {

// Patches per shared-memory row: tiles are at most 64 (FP64) or 128 cells wide.
constexpr int kPX = 34;

// Cells of a patch row: 16 bytes.
template <typename T>
constexpr int kW = 16 / static_cast<int>(sizeof(T));

// Tile of one launch (host-chosen, see plan_tile in poisson.cu).
struct Tile {
  int ix, iy;    // interior cells: ix a multiple of W up to W (kPX - 2), iy even
  int px, ey;    // extended tile: patches per row (ix / W + 2), rows
  int tx;        // tiles along x
  int chunk;     // k planes per block
};

// The cell that index c repeats, with the sign of a homogeneous-Dirichlet
// reflection.
__device__ __forceinline__ int image(int c, int n, int per, int dlo, int dhi, bool& neg) {
  neg = false;
  while(c < 0 || c >= n) {
    if(per) {
      c += c < 0 ? n : -n;
    } else if(c < 0) {
      c = -1 - c;
      neg ^= dlo != 0;
    } else {
      c = 2 * n - 1 - c;
      neg ^= dhi != 0;
    }
  }
  return c;
}

template <typename T>
struct Patch {
  T v[2][kW<T>];  // [row][x cell]
};

// The 16-byte vector of a patch row.
template <typename T>
using Vec = std::conditional_t<std::is_same_v<T, double>, double2, float4>;

template <typename T>
__device__ __forceinline__ void unpack(const Vec<T>& d, T (&v)[kW<T>]) {
  v[0] = d.x;
  v[1] = d.y;
  if constexpr(kW<T> == 4) {
    v[2] = d.z;
    v[3] = d.w;
  }
}

template <typename T>
__device__ __forceinline__ Vec<T> pack(const T (&v)[kW<T>]) {
  if constexpr(kW<T> == 4) return make_float4(v[0], v[1], v[2], v[3]);
  else return make_double2(v[0], v[1]);
}

// One thread's patch: image cells, signs, diagonal classes, interior flags
// (bit W r + c for cell c of row r).
template <typename T, bool SGN>
struct Place {
  static constexpr int W = kW<T>;
  static constexpr unsigned kAll = (1u << (2 * W)) - 1u;
  int p, row0;    // patch in its row, first extended row
  int xi[W];      // image columns
  int yj[2];      // image rows
  int off[2];     // offsets of the rows' first cells in a plane
  int yo[2];      // image rows times nx
  unsigned cls;   // diagonal classes of the cells (x + 4 y), four bits each
  unsigned neg;   // negated images
  unsigned in;    // interior cells of the domain
  int x0, y0;     // unmapped coordinates of the first cell
  bool vec;       // the row's cells are contiguous and 16-byte aligned

  __device__ __forceinline__ Place(const OpInfo& o, const Tile& t, int halo_rows) {
    p = threadIdx.x % t.px;
    row0 = 2 * (threadIdx.x / t.px);
    x0 = (blockIdx.x % t.tx) * t.ix + W * (p - 1);
    y0 = (blockIdx.x / t.tx) * t.iy + row0 - halo_rows;
    cls = 0;
    neg = 0;
    in = 0;
    bool nx_[W], ny_[2];
    vec = o.L.nx % W == 0;
#pragma unroll
    for(int c = 0; c < W; ++c) {
      xi[c] = image(x0 + c, o.L.nx, o.periodic[0], o.dir_lo[0], o.dir_hi[0], nx_[c]);
      vec = vec && xi[c] == xi[0] + c;
    }
    vec = vec && xi[0] % W == 0;
#pragma unroll
    for(int r = 0; r < 2; ++r) {
      yj[r] = image(y0 + r, o.L.ny, o.periodic[1], o.dir_lo[1], o.dir_hi[1], ny_[r]);
      yo[r] = yj[r] * o.L.nx;
      off[r] = yo[r] + xi[0];
    }
    const bool own = p > 0 && p < t.px - 1;
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < W; ++c) {
        const int e = row0 + r, bit = W * r + c;
        if(own && e >= halo_rows && e < t.ey - halo_rows && x0 + c < o.L.nx && y0 + r < o.L.ny)
          in |= 1u << bit;
        if(nx_[c] != ny_[r]) neg |= 1u << bit;
        cls |= static_cast<unsigned>(axis_class(xi[c], o.L.nx) + 4 * axis_class(yj[r], o.L.ny)) << (4 * bit);
      }
  }
  __device__ __forceinline__ bool interior(int r, int c) const { return (in >> (W * r + c)) & 1u; }

  // The patch of f's plane that starts at cell zo.
  __device__ __forceinline__ Patch<T> load(const T* __restrict__ f, int zo) const {
    Patch<T> q;
#pragma unroll
    for(int r = 0; r < 2; ++r) {
      if(vec) {
        unpack<T>(*reinterpret_cast<const Vec<T>*>(f + (zo + off[r])), q.v[r]);
      } else {
#pragma unroll
        for(int c = 0; c < W; ++c) q.v[r][c] = f[zo + yo[r] + xi[c]];
      }
    }
    return q;
  }

  // The same into the thread's own words of a ring slot (the block's threads
  // side by side, row by row), without waiting: take() reads them back.
  __device__ __forceinline__ void fetch(T* slot, const T* __restrict__ f, int zo) const {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(slot)) + 16 * threadIdx.x;
    const unsigned dr = 16 * blockDim.x;
    if(vec) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(f + (zo + off[0])) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + dr), "l"(f + (zo + off[1])) : "memory");
    } else {
      constexpr int w = sizeof(T);
#pragma unroll
      for(int c = 0; c < W; ++c) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + w * c), "l"(f + (zo + yo[0] + xi[c])), "n"(w) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + dr + w * c), "l"(f + (zo + yo[1] + xi[c])), "n"(w) : "memory");
      }
    }
  }

  __device__ __forceinline__ Patch<T> take(const T* slot) const {
    Patch<T> q;
    unpack<T>(*reinterpret_cast<const Vec<T>*>(slot + W * threadIdx.x), q.v[0]);
    unpack<T>(*reinterpret_cast<const Vec<T>*>(slot + W * (blockDim.x + threadIdx.x)), q.v[1]);
    return q;
  }

  // A loaded patch less the vector's pending mean (only problems without
  // Dirichlet faces have one) and with the signs of Dirichlet images.
  __device__ __forceinline__ void settle(Patch<T>& q, T shift, bool zneg) const {
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < W; ++c) {
        if constexpr(!SGN) q.v[r][c] -= shift;
        else if((((neg >> (W * r + c)) & 1u) != 0) != zneg) q.v[r][c] = -q.v[r][c];
      }
  }

  // Stores the interior cells into the plane that starts at cell zo.
  __device__ __forceinline__ void store(T* __restrict__ f, int zo, const Patch<T>& q) const {
    if(in == kAll && vec) {
      *reinterpret_cast<Vec<T>*>(f + (zo + off[0])) = pack<T>(q.v[0]);
      *reinterpret_cast<Vec<T>*>(f + (zo + off[1])) = pack<T>(q.v[1]);
    } else if(in != 0) {
#pragma unroll
      for(int c = 0; c < W; ++c) {
        if(interior(0, c)) f[zo + yo[0] + xi[c]] = q.v[0][c];
        if(interior(1, c)) f[zo + yo[1] + xi[c]] = q.v[1][c];
      }
    }
  }
};

// A field's plane in shared memory: ey rows of W runs of kPX cells, with a
// guard row before and after.  `me` is the thread's first cell.
template <typename T>
constexpr int kRow = kW<T> * kPX;

template <typename T>
__device__ __forceinline__ void publish(T* me, const Patch<T>& q) {
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int c = 0; c < kW<T>; ++c) me[r * kRow<T> + c * kPX] = q.v[r][c];
}

// Second differences along x and y of a published patch, each as the reference
// forms it (linsolve/poisson_solver.cpp:244-262): high - 2 centre + low.  For a
// smooth field the two operations are exact (what remains is a multiple of the
// values' last bit and small), so the operator's error is that of its value; as
// a multiple of the centre less the sums of the neighbours it would be that of
// the centre's term, larger by the square of the cells across the field, and A of
// a constant would not vanish.  At the rim of the extended tile the words read are
// not the true neighbours (another run's end, a guard row); the cells they spoil
// are never used: the halo shrinks by one cell per sweep.
template <typename T>
__device__ __forceinline__ T second_difference(T low, T centre, T high) {
  return (high - T(2) * centre) + low;
}

template <typename T>
__device__ __forceinline__ void differences(const T* me, const Patch<T>& q, Patch<T>& xs, Patch<T>& ys) {
  constexpr int W = kW<T>;
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int c = 0; c < W; ++c) {
      const T l = c > 0 ? q.v[r][c > 0 ? c - 1 : 0] : me[r * kRow<T> + (W - 1) * kPX - 1];
      const T h = c < W - 1 ? q.v[r][c < W - 1 ? c + 1 : 0] : me[r * kRow<T> + 1];
      xs.v[r][c] = second_difference(l, q.v[r][c], h);
    }
#pragma unroll
  for(int c = 0; c < W; ++c) {
    ys.v[0][c] = second_difference(me[c * kPX - kRow<T>], q.v[0][c], q.v[1][c]);
    ys.v[1][c] = second_difference(q.v[0][c], q.v[1][c], me[c * kPX + 2 * kRow<T>]);
  }
}

// Operator coefficients: A u = - ix (second difference along x) - iy (y) - iz (z).
// On a grid one cell deep (FLAT) the z term is zz u: its images are u itself, or
// -u at a Dirichlet face.
template <typename T>
struct Coef {
  T ix, iy, iz, zz;
  __device__ __forceinline__ explicit Coef(const OpInfo& o) {
    ix = T(o.inv2[0]);
    iy = T(o.inv2[1]);
    iz = T(o.inv2[2]);
    zz = T(o.periodic[2] ? 0.0 : 2.0 * o.inv2[2] * (o.dir_lo[2] + o.dir_hi[2]));
  }
};

// b - A u on a patch.
template <typename T, bool FLAT>
__device__ __forceinline__ Patch<T> residual(const Coef<T>& a, const Patch<T>& b, const Patch<T>& u,
                                             const Patch<T>& xs, const Patch<T>& ys, const Patch<T>& below,
                                             const Patch<T>& above) {
  Patch<T> o;
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int c = 0; c < kW<T>; ++c) {
      T t = b.v[r][c] + a.ix * xs.v[r][c];
      t += a.iy * ys.v[r][c];
      if constexpr(FLAT) t -= a.zz * u.v[r][c];
      else t += a.iz * second_difference(below.v[r][c], u.v[r][c], above.v[r][c]);
      o.v[r][c] = t;
    }
  return o;
}

// Threads of a march block: 512 at 128 registers fill an SM.
constexpr int kMaxThreads = 512;

// Planes streamed from memory pass through a ring of four slots per vector,
// copied asynchronously ahead of their use: with the loads in registers one
// plane ahead, waiting for them was the largest stall (28 % of the issue
// slots at 256^3), and registers for more there are none.
constexpr int kRing = 4;
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fetch_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Words of one published plane, its guard rows included, and of one ring
// slot; the shared memory of a kernel that streams `streams` vectors and
// publishes `fields` fields (two planes each): rings, planes, diagonal table.
// A grid one cell deep streams nothing and needs one plane per field.
// `parents`: room for the coarse correction's ring (k_ascend).
template <typename T>
__host__ __device__ inline int plane_words(const Tile& t) {
  return (t.ey + 2) * kRow<T>;
}
template <typename T>
__host__ __device__ inline int slot_words(const Tile& t) {
  return kW<T> * t.px * t.ey;
}
template <typename T>
inline size_t smem_bytes(const Tile& t, int streams, int fields, bool flat, bool parents = false) {
  if(flat) return (static_cast<size_t>(fields) * plane_words<T>(t) + 64) * sizeof(T);
  return (static_cast<size_t>(kRing) * streams * slot_words<T>(t) +
          static_cast<size_t>(2) * fields * plane_words<T>(t) + 64) * sizeof(T) +
         (parents ? static_cast<size_t>(kRing) * (t.px * t.ey / 2) * 8 : 0);
}

// The image plane of k, -2 <= k <= nz + 1 with nz >= 2, and whether it is a
// negated image.
__device__ __forceinline__ int zplane(const OpInfo& o, int k, bool& neg) {
  const int nz = o.L.nz;
  const bool lo = k < 0, hi = k >= nz;
  neg = (lo && o.dir_lo[2]) || (hi && o.dir_hi[2]);
  if(o.periodic[2]) return lo ? k + nz : hi ? k - nz : k;
  return lo ? -1 - k : hi ? 2 * nz - 1 - k : k;
}

// The image planes of consecutive k (from k >= 0), advanced without the case
// distinctions of zplane: the marching threads have no scalar unit to spare.
struct Walk {
  int k, kz, dk;
  __device__ __forceinline__ Walk(const OpInfo& o, int k_) : k(k_), dk(1) {
    bool neg;
    kz = zplane(o, k, neg);
    if(k >= o.L.nz && !o.periodic[2]) dk = -1;
  }
  __device__ __forceinline__ void next(const OpInfo& o) {
    ++k;
    kz += dk;
    if(k == o.L.nz) {
      if(o.periodic[2]) {
        kz = 0;
      } else {
        kz -= 1;
        dk = -1;
      }
    }
  }
};

__device__ __forceinline__ bool zneg(const OpInfo& o, int k) {
  return (k < 0 && o.dir_lo[2]) || (k >= o.L.nz && o.dir_hi[2]);
}

// omega / D on the planes of a march: the table is read again only when the z
// class changes.
template <typename T, bool CD>
struct Weights {
  const T* tab;
  Patch<T> w;
  int cz;
  __device__ __forceinline__ Weights(const T* t, T d0) : tab(t), cz(-1) {
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c) w.v[r][c] = d0;
  }
  __device__ __forceinline__ void at(const OpInfo& o, unsigned cls, int k) {
    if constexpr(!CD) {
      bool zn;
      const int z = axis_class(zplane(o, k, zn), o.L.nz);
      if(z == cz) return;
      cz = z;
#pragma unroll
      for(int r = 0; r < 2; ++r)
#pragma unroll
        for(int c = 0; c < kW<T>; ++c) w.v[r][c] = tab[((cls >> (4 * (kW<T> * r + c))) & 15u) + 16 * z];
    }
  }
};

template <typename T>
__device__ __forceinline__ Patch<T> times(const Patch<T>& w, const Patch<T>& u) {
  Patch<T> q;
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int c = 0; c < kW<T>; ++c) q.v[r][c] = w.v[r][c] * u.v[r][c];
  return q;
}

// u + w res: a damped Jacobi sweep from its residual.
template <typename T>
__device__ __forceinline__ Patch<T> relax(const Patch<T>& u, const Patch<T>& w, const Patch<T>& res) {
  Patch<T> q;
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int c = 0; c < kW<T>; ++c) q.v[r][c] = u.v[r][c] + w.v[r][c] * res.v[r][c];
  return q;
}

// Runs step(J, s) for s = s0 .. s1 with J = (s - s0) mod 4 a compile-time
// constant (the register slot of plane s).
template <typename Step>
__device__ __forceinline__ void ring4(int s0, int s1, Step step) {
  for(int s = s0; s <= s1; s += 4) {
    step(std::integral_constant<int, 0>(), s);
    if(s + 1 > s1) break;
    step(std::integral_constant<int, 1>(), s + 1);
    if(s + 2 > s1) break;
    step(std::integral_constant<int, 2>(), s + 2);
    if(s + 3 > s1) break;
    step(std::integral_constant<int, 3>(), s + 3);
  }
}

// Descent of one V-cycle level (v_cycle, linsolve/poisson_solver.cpp:597-624):
// both pre-sweeps from a zero correction, the residual and its restriction, in
// one pass over b:  a = omega b / D (pointwise), x = a + omega (b - A a) / D,
// bc = R (b - A x).  b carries the pending shift *sb_ptr (its mean, finest
// level).  The means the reference removes between these steps are constants
// (of a and x: A annihilates them, and the prolonged sum's constant is removed
// with mean(z)) or zero up to rounding (of bc: the residual of a zero-mean rhs
// has zero mean), so no sum is formed here.
//
// Bound: one read of b, one write of x and of bc (2.125 vectors); in FP64 at
// 256^3 the arithmetic and the shared-memory traffic are each near the DRAM time:
// 82 us (FP32 55), where the pre-sweeps and the residual with its restriction
// took 53 + 65 in two passes.
template <typename T, bool SGN, bool CD, bool FLAT>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_descend(OpInfo o, CLay oc, Tile t, const T* __restrict__ b, const double* sb_ptr, T* __restrict__ x,
              T* __restrict__ bc, int rx, int ry, int rz) {
  extern __shared__ __align__(16) unsigned char march_sm[];
  T* ring = reinterpret_cast<T*>(march_sm);
  const int sw = slot_words<T>(t), pw = plane_words<T>(t);
  T* planes = FLAT ? ring : ring + kRing * sw;
  T* tab = planes + (FLAT ? 2 : 4) * pw;
  if constexpr(!CD) {
    for(int q = threadIdx.x; q < 64; q += blockDim.x) tab[q] = T(2.0 / 3.0 * o.invd[q]);
    __syncthreads();
  }
  Weights<T, CD> W(tab, T(2.0 / 3.0 * o.invd[0]));
  const Place<T, SGN> pl(o, t, 2);
  const Coef<T> co(o);
  const T inv_children = T(1.0 / double(rx * ry * rz));
  const int nxy = o.L.nxy;
  const int k0 = blockIdx.y * t.chunk, k1 = min(k0 + t.chunk, o.L.nz);
  T* me = planes + (pl.row0 + 1) * kRow<T> + pl.p;  // field 0 of the even planes
  pdl_early();
  pdl_enter();
  const T sb = SGN ? T(0) : T(*sb_ptr);
  bool zn;
  Patch<T> racc;
  constexpr int PW = kW<T>;
  auto restrict_out = [&](int K) {
    if(pl.in == 0) return;
    if(rx == 2 && ry == 2) {
      T* out = bc + oc.idx(pl.x0 >> 1, pl.y0 >> 1, K);
#pragma unroll
      for(int c = 0; c < PW; c += 2)
        if(pl.interior(0, c))
          out[c / 2] = inv_children * ((racc.v[0][c] + racc.v[0][c + 1]) + (racc.v[1][c] + racc.v[1][c + 1]));
      return;
    }
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < PW; ++c) {
        if((ry == 2 && r == 1) || (rx == 2 && (c & 1)) || !pl.interior(r, c)) continue;
        T v = racc.v[r][c];
        if(rx == 2) v += racc.v[r][c | 1];
        if(ry == 2) v += racc.v[1][c];
        bc[oc.idx((pl.x0 + c) >> (rx - 1), (pl.y0 + r) >> (ry - 1), K)] = inv_children * v;
      }
  };
  Patch<T> xs, ys;
  if constexpr(FLAT) {
    Patch<T> bq = pl.load(b, 0);
    pl.settle(bq, sb, false);
    W.at(o, pl.cls, 0);
    const Patch<T> a = times(W.w, bq);
    publish(me, a);
    __syncthreads();
    differences(me, a, xs, ys);
    const Patch<T> xq = relax(a, W.w, residual<T, true>(co, bq, a, xs, ys, a, a));
    pl.store(x, 0, xq);
    publish(me + pw, xq);
    __syncthreads();
    differences(me + pw, xq, xs, ys);
    racc = residual<T, true>(co, bq, xq, xs, ys, xq, xq);
    restrict_out(0);
  } else {
    // step s: x(s) from a(s - 1 .. s + 1), then the residual of plane s - 1
    Patch<T> A[4], B[4], X[4];
    Walk f(o, k0);  // the next plane to fetch
    for(int q = 1; q <= 3; ++q) {
      if(f.k <= k1 + 1) pl.fetch(ring + (q & 3) * sw, b, f.kz * nxy);
      fetch_commit();
      f.next(o);
    }
    B[3] = pl.load(b, zplane(o, k0 - 2, zn) * nxy);
    pl.settle(B[3], sb, zn);
    W.at(o, pl.cls, k0 - 2);
    A[3] = times(W.w, B[3]);
    B[0] = pl.load(b, zplane(o, k0 - 1, zn) * nxy);
    pl.settle(B[0], sb, zn);
    W.at(o, pl.cls, k0 - 1);
    A[0] = times(W.w, B[0]);
    X[2] = X[3] = A[0];
    ring4(k0 - 1, k1, [&](auto jc, int s) {
      constexpr int J = jc, M = (J + 3) & 3, N = (J + 1) & 3, F = (J + 2) & 3;
      fetch_wait<2>();
      B[N] = pl.take(ring + N * sw);
      if(f.k <= k1 + 1) pl.fetch(ring + J * sw, b, f.kz * nxy);
      __syncwarp();
      fetch_commit();
      f.next(o);
      T* pa = me + (J & 1) * 2 * pw;
      publish(pa, A[J]);
      publish(pa + pw, X[M]);
      pl.settle(B[N], sb, SGN && zneg(o, s + 1));
      W.at(o, pl.cls, s + 1);
      A[N] = times(W.w, B[N]);
      __syncthreads();
      W.at(o, pl.cls, s);
      differences(pa, A[J], xs, ys);
      const Patch<T> xc = relax(A[J], W.w, residual<T, false>(co, B[J], A[J], xs, ys, A[M], A[N]));
      if(s >= k0 && s < k1) pl.store(x, s * nxy, xc);
      if(s > k0) {
        differences(pa + pw, X[M], xs, ys);
        const Patch<T> res = residual<T, false>(co, B[M], X[M], xs, ys, X[F], xc);
        const bool first = rz == 1 || ((s - 1) & 1) == 0;
#pragma unroll
        for(int r = 0; r < 2; ++r)
#pragma unroll
          for(int c = 0; c < kW<T>; ++c) racc.v[r][c] = first ? res.v[r][c] : racc.v[r][c] + res.v[r][c];
        if(rz == 1 || !first) restrict_out((s - 1) >> (rz - 1));
      }
      X[J] = xc;
      __syncwarp();
    });
  }
}

// Ascent of one V-cycle level (linsolve/poisson_solver.cpp:625-633): the
// coarse correction added and both post-sweeps, in one pass:  y = x + P e,
// y' = y + omega (b - A y) / D, out = y' + omega (b - A y') / D.  On the finest
// level (FINE) it also forms mean(out) and r.z for the CG; on the others no
// mean is needed (see k_descend).  sx, sy, sz: log2 of the coarsening ratios.
//
// Bound: reads x, b and e, writes out (3.125 vectors); 103 us at 256^3 in FP64 (71
// in FP32), where the prolongation with one sweep and the second sweep took 89 + 78.
template <typename T, bool SGN, bool CD, bool FLAT, bool FINE, bool PAIRS>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_ascend(OpInfo o, CLay lc, Tile t, const T* __restrict__ b, const double* sb_ptr, const T* __restrict__ x,
             const T* __restrict__ e, T* __restrict__ out, int sx, int sy, int sz, LevelScalars* ls,
             SolveScalars* sc, RedBuf rb) {
  extern __shared__ __align__(16) unsigned char march_sm[];
  T* ring = reinterpret_cast<T*>(march_sm);
  const int sw = slot_words<T>(t), pw = plane_words<T>(t);
  T* planes = FLAT ? ring : ring + kRing * 2 * sw;
  T* tab = planes + (FLAT ? 2 : 4) * pw;
  if constexpr(!CD) {
    for(int q = threadIdx.x; q < 64; q += blockDim.x) tab[q] = T(2.0 / 3.0 * o.invd[q]);
    __syncthreads();
  }
  Weights<T, CD> W(tab, T(2.0 / 3.0 * o.invd[0]));
  const Place<T, SGN> pl(o, t, 2);
  const Coef<T> co(o);
  const int nxy = o.L.nxy;
  const int k0 = blockIdx.y * t.chunk, k1 = min(k0 + t.chunk, o.L.nz);
  T* me = planes + (pl.row0 + 1) * kRow<T> + pl.p;
  pdl_early();
  pdl_enter();
  const T sb = SGN ? T(0) : T(*sb_ptr);
  bool zn;
  // the coarse correction of the patch: W / 2 parents (8 bytes) where both x
  // and y coarsen (PAIRS), streamed through a ring like x and b -- loaded into
  // registers two planes ahead they cost 18 us at 256^3 in FP64 and 18 of 84 in
  // FP32; else one per cell, loaded two planes ahead, always from valid cells
  // (under a condition the merge would wait for the load)
  constexpr int NR = PAIRS ? 1 : 2, NE = PAIRS ? kW<T> / 2 : kW<T>;
  struct Parents {
    T v[NR][NE];
  };
  T* ering = tab + 64;
  const int ew = PAIRS ? NE * blockDim.x : 0;
  const int e0 = lc.nx * (pl.yj[0] >> 1);
  auto lde = [&](int kz) {
    Parents q;
    const T* ep = e + lc.nxy * (kz >> sz);
#pragma unroll
    for(int r = 0; r < NR; ++r)
#pragma unroll
      for(int c = 0; c < NE; ++c)
        q.v[r][c] = PAIRS ? ep[e0 + (pl.xi[2 * c] >> 1)] : ep[lc.nx * (pl.yj[r] >> sy) + (pl.xi[c] >> sx)];
    return q;
  };
  auto fetch_e = [&](int slot, int kz) {
    const T* ep = e + (lc.nxy * (kz >> sz) + e0);
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(ering + slot * ew + NE * threadIdx.x));
    if(NE == 1 || pl.vec) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(ep + (pl.xi[0] >> 1)) : "memory");
    } else {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(ep + (pl.xi[0] >> 1)) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4), "l"(ep + (pl.xi[NE] >> 1)) : "memory");
    }
  };
  auto take_e = [&](int slot) {
    Parents q;
#pragma unroll
    for(int c = 0; c < NE; ++c) q.v[0][c] = ering[slot * ew + NE * threadIdx.x + c];
    return q;
  };
  // y = x + P e with the signs of Dirichlet images
  auto join = [&](Patch<T>& q, const Parents& ev, int k) {
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c) q.v[r][c] += PAIRS ? ev.v[0][c / 2] : ev.v[r % NR][c % NE];
    if constexpr(SGN) pl.settle(q, T(0), !FLAT && zneg(o, k));
  };
  double acc[2] = {0.0, 0.0};
  auto finish = [&](int k, const Patch<T>& v, const Patch<T>& bq) {
    pl.store(out, k * nxy, v);
    if constexpr(FINE) {
#pragma unroll
      for(int r = 0; r < 2; ++r)
#pragma unroll
        for(int c = 0; c < kW<T>; ++c)
          if(pl.interior(r, c)) {
            acc[0] += double(v.v[r][c]);
            acc[1] += double(bq.v[r][c]) * double(v.v[r][c]);
          }
    }
  };
  Patch<T> xs, ys;
  if constexpr(FLAT) {
    Patch<T> bq = pl.load(b, 0), y = pl.load(x, 0);
    pl.settle(bq, sb, false);
    join(y, lde(0), 0);
    W.at(o, pl.cls, 0);
    publish(me, y);
    __syncthreads();
    differences(me, y, xs, ys);
    const Patch<T> y1 = relax(y, W.w, residual<T, true>(co, bq, y, xs, ys, y, y));
    publish(me + pw, y1);
    __syncthreads();
    differences(me + pw, y1, xs, ys);
    finish(0, relax(y1, W.w, residual<T, true>(co, bq, y1, xs, ys, y1, y1)), bq);
  } else {
    // step s: y'(s) from y(s - 1 .. s + 1), then out(s - 1)
    Patch<T> Y[4], B[4], V[4];
    T* bring = ring + kRing * sw;
    // b is fetched a plane behind x: both are three steps ahead of their use
    int zb = zplane(o, k0 - 1, zn) * nxy;
    Walk f(o, k0);
    Parents E[4];
    for(int q = 1; q <= 3; ++q) {
      const int zx = f.kz * nxy;
      if(f.k <= k1 + 1) pl.fetch(ring + (q & 3) * sw, x, zx);
      if(f.k <= k1 + 1) pl.fetch(bring + (q - 1) * sw, b, zb);
      if constexpr(PAIRS) {
        if(f.k <= k1 + 1) fetch_e(q, f.kz);
      } else {
        if(q == 1) E[1] = lde(f.kz);
        if(q == 2) E[2] = lde(f.kz);
      }
      fetch_commit();
      zb = zx;
      f.next(o);
    }
    int ke = zplane(o, k0 + 2, zn);
    Y[3] = pl.load(x, zplane(o, k0 - 2, zn) * nxy);
    join(Y[3], lde(zplane(o, k0 - 2, zn)), k0 - 2);
    Y[0] = pl.load(x, zplane(o, k0 - 1, zn) * nxy);
    join(Y[0], lde(zplane(o, k0 - 1, zn)), k0 - 1);
    V[2] = V[3] = Y[0];
    B[3] = Y[0];
    ring4(k0 - 1, k1, [&](auto jc, int s) {
      constexpr int J = jc, M = (J + 3) & 3, N = (J + 1) & 3, F = (J + 2) & 3;
      fetch_wait<2>();
      Y[N] = pl.take(ring + N * sw);
      B[J] = pl.take(bring + J * sw);
      const int zx = f.kz * nxy;
      if constexpr(PAIRS) E[N] = take_e(N);
      if(f.k <= k1 + 1) pl.fetch(ring + J * sw, x, zx);       // plane s + 4
      if constexpr(PAIRS) {
        if(f.k <= k1 + 1) fetch_e(J, f.kz);
      }
      if(f.k <= k1 + 2) pl.fetch(bring + M * sw, b, zb);      // plane s + 3
      __syncwarp();
      fetch_commit();
      join(Y[N], E[N], s + 1);
      if constexpr(!PAIRS) E[M] = lde(ke);
      zb = zx;
      ke = max(0, min(f.kz, o.L.nz - 1));
      f.next(o);
      T* pa = me + (J & 1) * 2 * pw;
      publish(pa, Y[J]);
      publish(pa + pw, V[M]);
      pl.settle(B[J], sb, SGN && zneg(o, s));
      __syncthreads();
      W.at(o, pl.cls, s);
      differences(pa, Y[J], xs, ys);
      const Patch<T> vc = relax(Y[J], W.w, residual<T, false>(co, B[J], Y[J], xs, ys, Y[M], Y[N]));
      if(s > k0) {
        W.at(o, pl.cls, s - 1);
        differences(pa + pw, V[M], xs, ys);
        finish(s - 1, relax(V[M], W.w, residual<T, false>(co, B[M], V[M], xs, ys, V[F], vc)), B[M]);
      }
      V[J] = vc;
      __syncwarp();
    });
  }
  if constexpr(FINE) {
    const bool mx[2] = {false, false};
    reduce_finish<2>(acc, mx, rb, [=](const Sums<2>& s) {
      const double mean = sc->zero_mean ? s.v[0] / sc->n : 0.0;
      ls->sx = mean;
      // r.z with z = out - mean (linsolve/poisson_solver.cpp:749, :791)
      const double rz_new = s.v[1] - mean * (sc->sum_r - sc->n * sc->sr);
      if(!sc->first) sc->beta = rz_new / sc->rz;
      sc->rz = rz_new;
    });
  }
}


constexpr double kBreakdown = 1.0e-30;  // linsolve/poisson_solver.cpp:757

// The buffers of the search direction: an iteration reads one and writes the
// other (a tile's halo still needs the old values when its neighbour writes).
template <typename T>
struct Direction {
  T* p[2];
};

// New search direction and its products (linsolve/poisson_solver.cpp:750-761):
// p = (z - sz) + beta p (first iteration: z - sz) and p.Ap; A p itself is not
// stored -- k_advance forms it again from p, which costs its nine operations
// instead of a vector written and read back.  The means of p and A p that the
// reference removes are zero up to rounding (z - sz has none, A annihilates
// constants) and are left in; those of x and of the residual, which they would
// move, are removed every iteration.  Bound: reads z and p, writes p (3 vectors); at
// 256^3 72 us in FP64, where the separate p update and A p took 71 + 66.
template <typename T, bool SGN, bool FLAT>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_direction(OpInfo o, Tile t, const T* __restrict__ z, const LevelScalars* ls0, Direction<T> d,
                SolveScalars* sc, RedBuf rb) {
  extern __shared__ __align__(16) unsigned char march_sm[];
  T* ring = reinterpret_cast<T*>(march_sm);
  const int sw = slot_words<T>(t), pw = plane_words<T>(t);
  T* pring = ring + kRing * sw;
  const Place<T, SGN> pl(o, t, 1);
  const Coef<T> co(o);
  const int nxy = o.L.nxy;
  const int k0 = blockIdx.y * t.chunk, k1 = min(k0 + t.chunk, o.L.nz);
  T* me = (FLAT ? ring : ring + 2 * kRing * sw) + (pl.row0 + 1) * kRow<T> + pl.p;
  pdl_early();
  pdl_enter();
  const bool first = sc->first != 0;
  const int turn = sc->body_runs & 1;
  const T* __restrict__ po = d.p[turn ^ 1];
  T* __restrict__ pn = d.p[turn];
  const T sz = SGN ? T(0) : T(ls0->sx);
  const T beta = first ? T(0) : T(sc->beta);
  double acc[1] = {0.0};
  auto combine = [&](Patch<T>& q, const Patch<T>& old, bool zn) {
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c) {
        const T zv = q.v[r][c] - sz;
        q.v[r][c] = first ? zv : zv + beta * old.v[r][c];
      }
    if constexpr(SGN) pl.settle(q, T(0), zn);
  };
  auto point = [&](int k, const Patch<T>& v, const Patch<T>& minus_av) {
    pl.store(pn, k * nxy, v);
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c)
        if(pl.interior(r, c)) acc[0] -= double(v.v[r][c]) * double(minus_av.v[r][c]);
  };
  const Patch<T> none = {};
  Patch<T> xs, ys;
  bool zn;
  if constexpr(FLAT) {
    Patch<T> q = pl.load(z, 0);
    combine(q, first ? none : pl.load(po, 0), false);
    publish(me, q);
    __syncthreads();
    differences(me, q, xs, ys);
    point(0, q, residual<T, true>(co, none, q, xs, ys, q, q));
  } else {
    // step s: p(s + 1) is combined, A p(s) formed
    Patch<T> P[4];
    Walk f(o, k0 + 1);
    for(int q = 1; q <= 3; ++q) {
      if(f.k <= k1) {
        pl.fetch(ring + (q & 3) * sw, z, f.kz * nxy);
        pl.fetch(pring + (q & 3) * sw, po, f.kz * nxy);
      }
      fetch_commit();
      f.next(o);
    }
    P[3] = pl.load(z, zplane(o, k0 - 1, zn) * nxy);
    combine(P[3], pl.load(po, zplane(o, k0 - 1, zn) * nxy), zn);
    P[0] = pl.load(z, k0 * nxy);
    combine(P[0], pl.load(po, k0 * nxy), false);
    ring4(k0, k1 - 1, [&](auto jc, int s) {
      constexpr int J = jc, M = (J + 3) & 3, N = (J + 1) & 3;
      fetch_wait<2>();
      P[N] = pl.take(ring + N * sw);
      const Patch<T> old = pl.take(pring + N * sw);
      if(f.k <= k1) {  // plane s + 4
        pl.fetch(ring + J * sw, z, f.kz * nxy);
        pl.fetch(pring + J * sw, po, f.kz * nxy);
      }
      __syncwarp();
      fetch_commit();
      f.next(o);
      T* pa = me + (J & 1) * pw;
      publish(pa, P[J]);
      combine(P[N], old, SGN && zneg(o, s + 1));
      __syncthreads();
      differences(pa, P[J], xs, ys);
      point(s, P[J], residual<T, false>(co, none, P[J], xs, ys, P[M], P[N]));
      __syncwarp();
    });
  }
  const bool mx[1] = {false};
  reduce_finish<1>(acc, mx, rb, [=](const Sums<1>& s) {
    sc->first = 0;
    sc->pap = s.v[0];
    if(fabs(s.v[0]) < kBreakdown) sc->stop = 1;
    else sc->alpha = sc->rz / s.v[0];
  });
}

// Solution and residual update (linsolve/poisson_solver.cpp:762-782):
// x = (x - sx) + alpha p, r = (r - sr) - alpha A p (in FP64 arithmetic), the
// residual's norm and the convergence test, and the means of the new x and r (a
// large mean in the initial guess leaves its rounding in the first x).  Bound:
// reads p, x and r, writes x and r (5 vectors); at 256^3 119 to 122 us in FP64,
// where the update from a stored A p took 142.
template <typename T, bool SGN, bool FLAT>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_advance(OpInfo o, Tile t, Direction<T> d, T* __restrict__ x, T* __restrict__ r, SolveScalars* sc, RedBuf rb,
              cudaGraphConditionalHandle cond) {
  extern __shared__ __align__(16) unsigned char march_sm[];
  T* ring = reinterpret_cast<T*>(march_sm);
  const int sw = slot_words<T>(t), pw = plane_words<T>(t);
  T *xring = ring + kRing * sw, *rring = xring + kRing * sw;
  const Place<T, SGN> pl(o, t, 1);
  const Coef<T> co(o);
  const int nxy = o.L.nxy;
  const int k0 = blockIdx.y * t.chunk, k1 = min(k0 + t.chunk, o.L.nz);
  T* me = (FLAT ? ring : rring + kRing * sw) + (pl.row0 + 1) * kRow<T> + pl.p;
  pdl_early();
  pdl_enter();
  const int stop = sc->stop;
  const T* __restrict__ p = d.p[sc->body_runs & 1];
  const double alpha = sc->alpha, sr = sc->sr;
  const T sx = T(sc->sx), ax = T(alpha);
  double acc[3] = {0.0, 0.0, 0.0};
  auto point = [&](int k, const Patch<T>& pv, const Patch<T>& minus_av, const Patch<T>& xv, const Patch<T>& rv) {
    Patch<T> xn, rn;
#pragma unroll
    for(int q = 0; q < 2; ++q)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c) {
        const double vr = (double(rv.v[q][c]) - sr) + alpha * double(minus_av.v[q][c]);
        xn.v[q][c] = (xv.v[q][c] - sx) + ax * pv.v[q][c];
        rn.v[q][c] = T(vr);
        if(pl.interior(q, c)) {
          acc[0] += vr;
          acc[1] += vr * vr;
          if constexpr(!SGN) acc[2] += double(xn.v[q][c]);
        }
      }
    pl.store(x, k * nxy, xn);
    pl.store(r, k * nxy, rn);
  };
  const Patch<T> none = {};
  Patch<T> xs, ys;
  bool zn;
  if(stop) {
  } else if constexpr(FLAT) {
    Patch<T> q = pl.load(p, 0);
    if constexpr(SGN) pl.settle(q, T(0), false);
    publish(me, q);
    const Patch<T> xv = pl.load(x, 0), rv = pl.load(r, 0);
    __syncthreads();
    differences(me, q, xs, ys);
    point(0, q, residual<T, true>(co, none, q, xs, ys, q, q), xv, rv);
  } else {
    // step s: plane s; p three planes ahead, x and r (own cells only) likewise
    Patch<T> P[4];
    int zo = k0 * nxy;
    Walk f(o, k0 + 1);
    for(int q = 1; q <= 3; ++q) {
      const int zp = f.kz * nxy;
      if(f.k <= k1) pl.fetch(ring + (q & 3) * sw, p, zp);
      if(f.k <= k1 && pl.in != 0) {
        pl.fetch(xring + (q - 1) * sw, x, zo);
        pl.fetch(rring + (q - 1) * sw, r, zo);
      }
      fetch_commit();
      zo = zp;
      f.next(o);
    }
    P[3] = pl.load(p, zplane(o, k0 - 1, zn) * nxy);
    if constexpr(SGN) pl.settle(P[3], T(0), zn);
    P[0] = pl.load(p, k0 * nxy);
    if constexpr(SGN) pl.settle(P[0], T(0), false);
    ring4(k0, k1 - 1, [&](auto jc, int s) {
      constexpr int J = jc, M = (J + 3) & 3, N = (J + 1) & 3;
      fetch_wait<2>();
      P[N] = pl.take(ring + N * sw);
      const int zp = f.kz * nxy;
      if(f.k <= k1) pl.fetch(ring + J * sw, p, zp);  // plane s + 4
      if(f.k <= k1 && pl.in != 0) {                  // plane s + 3
        pl.fetch(xring + M * sw, x, zo);
        pl.fetch(rring + M * sw, r, zo);
      }
      __syncwarp();
      fetch_commit();
      zo = zp;
      f.next(o);
      T* pa = me + (J & 1) * pw;
      publish(pa, P[J]);
      if constexpr(SGN) pl.settle(P[N], T(0), zneg(o, s + 1));
      __syncthreads();
      differences(pa, P[J], xs, ys);
      point(s, P[J], residual<T, false>(co, none, P[J], xs, ys, P[M], P[N]), pl.take(xring + J * sw),
            pl.take(rring + J * sw));
      __syncwarp();
    });
  }
  const bool mx[3] = {false, false, false};
  reduce_finish<3>(acc, mx, rb, [=](const Sums<3>& s) {
    sc->body_runs += 1;
    if(sc->stop) {
      sc->cont = 0;
      if(cond) cudaGraphSetConditional(cond, 0);
      return;
    }
    const int n = sc->n;
    const int zm = sc->zero_mean;
    sc->sx = zm ? s.v[2] / n : 0.0;
    const double srn = zm ? s.v[0] / n : 0.0;
    sc->sr = srn;
    sc->sum_r = s.v[0];
    const double ss = fmax(s.v[1] - n * srn * srn, 0.0);
    sc->rnorm = sqrt(ss / n);
    sc->iterations += 1;
    sc->rel = sc->r0 > 0.0 ? sc->rnorm / sc->r0 : 0.0;
    if(sc->rel <= sc->tol) sc->converged = 1;
    if(sc->hist != nullptr && sc->iterations < sc->hist_cap) sc->hist[sc->iterations] = sc->rnorm;
    // the reference's loop: at most max_iterations iterations, stop on convergence
    sc->cont = (sc->converged || sc->iterations >= sc->max_it) ? 0 : 1;
    if(cond) cudaGraphSetConditional(cond, sc->cont);
  });
}


// What a solve starts with; see start_solve.
struct SolveStart {
  double tol;
  int max_it, n, zero_mean;
  double* hist;
  int hist_cap;
};

// The scalars of a new solve from its residual's sum and sum of squares
// (linsolve/poisson_solver.cpp:717-739).
__device__ __forceinline__ void start_solve(SolveScalars* sc, const SolveStart& a, double sum, double squares) {
  if(!a.zero_mean) {
    sc->sb = 0.0;
    sc->sx = 0.0;
    sc->removed_rhs_mean = 0.0;
  }
  const double sr = a.zero_mean ? sum / a.n : 0.0;
  const double r0 = sqrt(fmax(squares - a.n * sr * sr, 0.0) / a.n);
  sc->zero_mean = a.zero_mean;
  sc->n = a.n;
  sc->tol = a.tol;
  sc->max_it = a.max_it;
  sc->hist = a.hist;
  sc->hist_cap = a.hist_cap;
  sc->outer = 0;
  sc->sr = sr;
  sc->sum_r = sum;
  sc->r0 = r0;
  sc->rnorm = r0;
  sc->iterations = 0;
  sc->stop = 0;
  sc->converged = r0 <= a.tol ? 1 : 0;
  sc->rel = sc->converged || r0 <= 0.0 ? 0.0 : 1.0;
  sc->first = 1;
  sc->body_runs = 0;
  sc->cont = sc->converged ? 0 : 1;
  if(a.hist != nullptr && a.hist_cap > 0) a.hist[0] = r0;
}

// The residual r = (b - sb) - A (x - sx) in FP64.  START: of the initial guess,
// beginning a solve; else of the mixed path's corrected solution: its norm, the
// convergence test and the outer loop's control (si: the inner solve's scalars).
// Bound: reads x and b, writes r (3 vectors); the column kernel it replaces took
// 125 us at 256^3.
template <bool SGN, bool FLAT, bool START>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_residual(OpInfo o, Tile t, const double* __restrict__ x, const double* __restrict__ b,
               double* __restrict__ res, SolveScalars* sc, const SolveScalars* si, SolveStart start, RedBuf rb) {
  using T = double;
  extern __shared__ __align__(16) unsigned char march_sm[];
  T* ring = reinterpret_cast<T*>(march_sm);
  const int sw = slot_words<T>(t), pw = plane_words<T>(t);
  T* bring = ring + kRing * sw;
  const Place<T, SGN> pl(o, t, 1);
  const Coef<T> co(o);
  const int nxy = o.L.nxy;
  const int k0 = blockIdx.y * t.chunk, k1 = min(k0 + t.chunk, o.L.nz);
  T* me = (FLAT ? ring : bring + kRing * sw) + (pl.row0 + 1) * kRow<T> + pl.p;
  pdl_early();
  pdl_enter();
  const T sb = SGN ? 0.0 : sc->sb, sx = SGN ? 0.0 : sc->sx;
  double acc[2] = {0.0, 0.0};
  auto point = [&](int k, const Patch<T>& v) {
    pl.store(res, k * nxy, v);
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c)
        if(pl.interior(r, c)) {
          acc[0] += v.v[r][c];
          acc[1] += v.v[r][c] * v.v[r][c];
        }
  };
  auto centred = [&](Patch<T> q) {
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int c = 0; c < kW<T>; ++c) q.v[r][c] -= sb;
    return q;
  };
  Patch<T> xs, ys;
  bool zn;
  if constexpr(FLAT) {
    Patch<T> q = pl.load(x, 0);
    pl.settle(q, sx, false);
    publish(me, q);
    const Patch<T> bq = centred(pl.load(b, 0));
    __syncthreads();
    differences(me, q, xs, ys);
    point(0, residual<T, true>(co, bq, q, xs, ys, q, q));
  } else {
    Patch<T> X[4];
    int zo = k0 * nxy;
    Walk f(o, k0 + 1);
    for(int q = 1; q <= 3; ++q) {
      const int zx = f.kz * nxy;
      if(f.k <= k1) pl.fetch(ring + (q & 3) * sw, x, zx);
      if(f.k <= k1 && pl.in != 0) pl.fetch(bring + (q - 1) * sw, b, zo);
      fetch_commit();
      zo = zx;
      f.next(o);
    }
    X[3] = pl.load(x, zplane(o, k0 - 1, zn) * nxy);
    pl.settle(X[3], sx, zn);
    X[0] = pl.load(x, k0 * nxy);
    pl.settle(X[0], sx, false);
    ring4(k0, k1 - 1, [&](auto jc, int s) {
      constexpr int J = jc, M = (J + 3) & 3, N = (J + 1) & 3;
      fetch_wait<2>();
      X[N] = pl.take(ring + N * sw);
      const int zx = f.kz * nxy;
      if(f.k <= k1) pl.fetch(ring + J * sw, x, zx);                  // plane s + 4
      if(f.k <= k1 && pl.in != 0) pl.fetch(bring + M * sw, b, zo);   // plane s + 3
      __syncwarp();
      fetch_commit();
      zo = zx;
      f.next(o);
      T* pa = me + (J & 1) * pw;
      publish(pa, X[J]);
      pl.settle(X[N], sx, SGN && zneg(o, s + 1));
      __syncthreads();
      differences(pa, X[J], xs, ys);
      point(s, residual<T, false>(co, centred(pl.take(bring + J * sw)), X[J], xs, ys, X[M], X[N]));
      __syncwarp();
    });
  }
  const bool mx[2] = {false, false};
  reduce_finish<2>(acc, mx, rb, [=](const Sums<2>& s) {
    if constexpr(START) {
      start_solve(sc, start, s.v[0], s.v[1]);
    } else {
      const int n = sc->n;
      const double sr = sc->zero_mean ? s.v[0] / n : 0.0;
      sc->sr = sr;
      sc->sum_r = s.v[0];
      const double rn = sqrt(fmax(s.v[1] - n * sr * sr, 0.0) / n);
      sc->rnorm = rn;
      sc->iterations += si->iterations;
      sc->body_runs += si->body_runs;
      sc->outer += 1;
      sc->rel = sc->r0 > 0.0 ? rn / sc->r0 : 0.0;
      if(sc->rel <= sc->tol) sc->converged = 1;
      if(sc->hist != nullptr && sc->outer < sc->hist_cap) sc->hist[sc->outer] = rn;
      const bool stalled = si->iterations == 0;
      sc->cont = (sc->converged || sc->iterations >= sc->max_it || sc->outer >= 100 || stalled) ? 0 : 1;
    }
  });
}

}  // namespace march
}  // namespace ofb
