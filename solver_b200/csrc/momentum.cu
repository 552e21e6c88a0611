// Momentum-side stencils: the TVD/van Leer advection term, the rest of the
// predictor right-hand side (diffusion, pressure gradient, factorisation
// correction and the AB2 combination in one pass), each one launch for the three
// components, and the Taylor-Green initial state.
#include "kernels.hpp"
#include "quotient.cuh"

namespace ofb {

namespace {

constexpr double kSmallDenominator = 1.0e-14;  // solver/momentum_terms.cpp:14

// n / d as the division rounds it, within quotient_in_range (quotient.cuh).  The
// hardware's reciprocal approximation reads the upper half of d and gives the
// upper half of the result (20 fraction bits each: relative error below 2^-19).
__device__ __forceinline__ double quotient(double n, double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  return quotient_from(n, d, r);
}

// Branch-free form of one reconstruct_face call: every candidate value is
// loaded before the velocity sign is known and the reference's three cases
// (first-order upwind for |u_f| < 1e-14 or near the storage bounds, van Leer
// MUSCL otherwise; solver/momentum_terms.cpp:42-151) are chosen by selects.
// EXACT: with the division itself; else `past` is set where quotient() is outside
// its range.
template <bool EXACT>
__device__ __forceinline__ double tvd_face(double vel, double left, double right, double far_left,
                                           bool far_left_ok, double far_right, bool far_right_ok, bool& past) {
  const bool up = vel >= 0.0;
  const double delta = right - left;
  const double num = up ? left - far_left : far_right - right;
  // safe_ratio and limiter_value (solver/momentum_terms.cpp:26-40) enter as
  // 0.5 phi(r) delta with r = num / delta (0 when |delta| < 1e-14) and
  // phi = (r + |r|) / (1 + |r|): zero unless r > 0, and then equal to
  // num delta / (delta + num) -- one division instead of two; the value
  // differs from the two-division form by rounding only (r > 0 is read off
  // the product num delta, whose underflow stands for a value below 1e-290).
  const double nd = num * delta;
  // (comparisons that let a NaN through, as the reference's formula does)
  const bool positive = !(fabs(delta) < kSmallDenominator) && !(nd <= 0.0);
  const double den = delta + num;
  double half_phi_delta;
  if constexpr(EXACT) {
    half_phi_delta = positive ? nd / den : 0.0;
  } else {
    half_phi_delta = positive ? quotient(nd, den) : 0.0;
    past = past || (positive && !quotient_in_range(__double2hiint(nd), __double2hiint(den), __double2loint(den)));
  }
  const double muscl = up ? left + half_phi_delta : right - half_phi_delta;
  const bool first_order = fabs(vel) < kSmallDenominator || (up ? !far_left_ok : !far_right_ok);
  return first_order ? (up ? left : right) : muscl;
}

// The three components of one launch: consecutive blocks take the same tile
// of u, v and w, which read the same velocity cells (from L2), and a step of a
// small grid is one launch instead of three.  Extents are the largest
// component's; a block clips to its own.
struct Tile3 {
  int comp, bx;
};
__device__ __forceinline__ Tile3 component_tile() {
  return Tile3{static_cast<int>(blockIdx.x % 3), static_cast<int>(blockIdx.x / 3)};
}

// The limited value carried by the face between storage points q - st and q
// of f (position pd along the axis, smax its last storage index), times the
// face's velocity (compute_{u,v,w}_advection, solver/momentum_terms.cpp:153-266).
template <bool EXACT>
__device__ __forceinline__ double face_flux(double vel, double fm1, double f0, double fm2, bool fm2_ok, double fp1,
                                            bool fp1_ok, bool& past) {
  return vel * tvd_face<EXACT>(vel, fm1, f0, fm2, fm2_ok, fp1, fp1_ok, past);
}

// Advection term of component C at the active points of a tile.  A point's
// upper face is its neighbour's lower one: along x it comes from the next lane
// (a warp evaluates 32 faces for 31 points), along z from the thread's next
// plane; only y faces are evaluated twice -- four faces per point instead of
// six, each the same operations as before (at 256^3 606 instead of 755 us when
// that was changed, at four blocks per SM; three 690, five 616).
//
// Returns whether a limiter's quotient was outside the fast form's range; the
// warp's points are then formed again with the division.  At 256^3 659 us; a
// division in every face takes 735, a branch to it at every face 730, the
// nearly always correct quotient that this replaces took 605.
constexpr int kAdvectTile = kTX - 1;

template <int C, bool EXACT>
__device__ __forceinline__ bool advect_tile(const Grid& g, const double* __restrict__ u,
                                            const double* __restrict__ v, const double* __restrict__ w,
                                            double* __restrict__ out, int bx, int kchunk) {
  bool past = false;
  const double* __restrict__ vel[3] = {u, v, w};
  const double* __restrict__ f = vel[C];
  const Lay L = make_lay(g, kFaceX + C);
  // lanes past the end repeat the last face so that every lane can exchange
  const int ip = bx * kAdvectTile + threadIdx.x + 1, jp = blockIdx.y * kTY + threadIdx.y + 1;
  const int i = min(ip, L.nx + 1), j = min(jp, L.ny);
  const bool own = threadIdx.x < kAdvectTile && ip <= L.nx && jp <= L.ny;
  const int k0 = blockIdx.z * kchunk + 1;
  const int k1 = min(k0 + kchunk, L.nz + 1);
  if(k0 >= k1) return false;
  const double ihx = 1.0 / g.dx, ihy = 1.0 / g.dy, ihz = 1.0 / g.dz;
  int q = L.idx(i, j, k0);
  // velocity component d at this component's point: the mean of its two values
  // there (d != C), at storage offsets b and a
  auto at = [&](int d, int k, int& a, int& b) {
    const Lay D = make_lay(g, kFaceX + d);
    a = D.idx(i, j, k);
    b = a - D.stride(C);
  };
  double zm1 = f[q - L.sxy], z0 = f[q], zp1 = f[q + L.sxy];
  double zlo;  // flux through the lower z face
  {
    double vz;
    if(C == 2) {
      vz = 0.5 * (zm1 + z0);
    } else {
      int a, b;
      at(2, k0, a, b);
      vz = 0.5 * (w[b] + w[a]);
    }
    zlo = face_flux<EXACT>(vz, zm1, z0, f[k0 >= 2 ? q - 2 * L.sxy : q - L.sxy], k0 >= 2, zp1, k0 + 1 <= L.sz - 1, past);
  }
  for(int k = k0; k < k1; ++k, q += L.sxy) {
    // x: this point's lower face, the upper one from the next lane
    double flux;
    {
      const double fm1 = f[q - 1], fp1 = f[i + 1 <= L.sx - 1 ? q + 1 : q];
      const double fm2 = f[i >= 2 ? q - 2 : q - 1];
      double vx;
      if(C == 0) {
        vx = 0.5 * (fm1 + z0);
      } else {
        int a, b;
        at(0, k, a, b);
        vx = 0.5 * (u[b] + u[a]);
      }
      const double lo = face_flux<EXACT>(vx, fm1, z0, fm2, i >= 2, fp1, i + 1 <= L.sx - 1, past);
      flux = (__shfl_down_sync(0xffffffffu, lo, 1) - lo) * ihx;
    }
    // y: both faces
    {
      const double fm1 = f[q - L.sx], fp1 = f[q + L.sx];
      const double fm2 = f[j >= 2 ? q - 2 * L.sx : q - L.sx], fp2 = f[j + 2 <= L.sy - 1 ? q + 2 * L.sx : q + L.sx];
      double vl, vh;
      if(C == 1) {
        vl = 0.5 * (fm1 + z0);
        vh = 0.5 * (z0 + fp1);
      } else {
        int a, b;
        at(1, k, a, b);
        const int sd = make_lay(g, kFaceY).sx;
        vl = 0.5 * (v[b] + v[a]);
        vh = 0.5 * (v[b + sd] + v[a + sd]);
      }
      flux += (face_flux<EXACT>(vh, z0, fp1, fm1, true, fp2, j + 2 <= L.sy - 1, past) -
               face_flux<EXACT>(vl, fm1, z0, fm2, j >= 2, fp1, true, past)) * ihy;
    }
    // z: the upper face, kept for the next plane
    {
      const double zp2 = f[k + 2 <= L.sz - 1 ? q + 2 * L.sxy : q + L.sxy];
      double vz;
      if(C == 2) {
        vz = 0.5 * (z0 + zp1);
      } else {
        int a, b;
        at(2, k + 1, a, b);
        vz = 0.5 * (w[b] + w[a]);
      }
      const double zhi = face_flux<EXACT>(vz, z0, zp1, zm1, true, zp2, k + 2 <= L.sz - 1, past);
      flux += (zhi - zlo) * ihz;
      zlo = zhi;
      zm1 = z0;
      z0 = zp1;
      zp1 = zp2;
    }
    if(own) out[q] = flux;
  }
  return past;
}

// Advection term of every component at its active points (the first half of
// assemble_predictor_rhs, solver/taylor_green.cpp:238).  Bound by its issue
// slots (the limiter's selects and FP64 operations).
__global__ void __launch_bounds__(kTX* kTY, 4)
    k_advect_bf(Grid g, const double* __restrict__ u, const double* __restrict__ v,
                const double* __restrict__ w, double* __restrict__ au, double* __restrict__ av,
                double* __restrict__ aw, int kchunk) {
  const Tile3 t = component_tile();
  if(t.comp == 0) {
    if(__any_sync(0xffffffffu, advect_tile<0, false>(g, u, v, w, au, t.bx, kchunk)))
      advect_tile<0, true>(g, u, v, w, au, t.bx, kchunk);
  } else if(t.comp == 1) {
    if(__any_sync(0xffffffffu, advect_tile<1, false>(g, u, v, w, av, t.bx, kchunk)))
      advect_tile<1, true>(g, u, v, w, av, t.bx, kchunk);
  } else {
    if(__any_sync(0xffffffffu, advect_tile<2, false>(g, u, v, w, aw, t.bx, kchunk)))
      advect_tile<2, true>(g, u, v, w, aw, t.bx, kchunk);
  }
}

// Blocks of k_advect_bf: as launch3_components, on tiles of kAdvectTile points.
Launch3 launch3_advection(const Grid& g) {
  Launch3 l = launch3_components(g);
  l.grid.x = 3 * ((g.nx + 1 + kAdvectTile - 1) / kAdvectTile);
  return l;
}

// What one plane contributes to the predictor at a point: the value and its
// second differences in x, in y and in both.
struct PlaneTerms {
  double c, xx, yy, xy;
};

__device__ __forceinline__ PlaneTerms plane_terms(const double* __restrict__ f, int q, int sx, double ix,
                                                  double iy) {
  double m[3][3];
#pragma unroll
  for(int b = 0; b < 3; ++b)
#pragma unroll
    for(int e = 0; e < 3; ++e) m[b][e] = f[q + (e - 1) + (b - 1) * sx];
  double d[3];
#pragma unroll
  for(int b = 0; b < 3; ++b) d[b] = (m[b][2] - 2.0 * m[b][1] + m[b][0]) * ix;
  return PlaneTerms{m[1][1], d[1], (m[2][1] - 2.0 * m[1][1] + m[0][1]) * iy, (d[2] - 2.0 * d[1] + d[0]) * iy};
}

// The rest of assemble_predictor_rhs (solver/taylor_green.cpp:239-255):
// diffusion, total-pressure gradient, factorisation correction and the AB2
// combination with the advection term computed by k_advect_bf.  A thread
// marches k with the terms of three planes in registers: the 27-point
// correction is the z second difference of the planes' xx, yy and xy, so a
// point loads the nine cells of one new plane instead of 27.
template <int C>
__device__ __forceinline__ void predictor_tile(const PredictorArgs& a, int bx, int kchunk) {
  const Grid& g = a.g;
  const Lay L = make_lay(g, kFaceX + C);
  const Lay P = make_lay(g, kCell);
  const int i = bx * kTX + threadIdx.x + 1;
  const int j = blockIdx.y * kTY + threadIdx.y + 1;
  if(i > L.nx || j > L.ny) return;
  const int k0 = blockIdx.z * kchunk + 1;
  const int k1 = min(k0 + kchunk, L.nz + 1);
  if(k0 >= k1) return;
  const double ih = 1.0 / g.h(C);
  const double ix = 1.0 / (g.dx * g.dx), iy = 1.0 / (g.dy * g.dy), iz = 1.0 / (g.dz * g.dz);
  const bool three_d = a.variant != 1 && g.nz != 1;
  const double s_gp = -a.dt;
  const double s_dif = 0.5 * a.dt * a.nu;
  const double s_adv = a.has_prev ? -1.5 * a.dt : -a.dt;
  const double s_prev = 0.5 * a.dt;
  const double s_corr = a.alpha * a.alpha;
  const double* __restrict__ f = a.cur[C];
  const double* __restrict__ p = a.p;
  const int pstC = P.stride(C);
  int q = L.idx(i, j, k0);
  PlaneTerms lo = plane_terms(f, q - L.sxy, L.sx, ix, iy), mid = plane_terms(f, q, L.sx, ix, iy);
  for(int k = k0; k < k1; ++k, q += L.sxy) {
    const PlaneTerms hi = plane_terms(f, q + L.sxy, L.sx, ix, iy);
    const int pq = P.idx(i, j, k);
    const double gp = (p[pq] - p[pq - pstC]) * ih;
    const double adv = a.adv[C][q];
    const double prev = a.has_prev ? a.prev[C][q] : 0.0;
    const double lap = mid.xx + mid.yy + (hi.c - 2.0 * mid.c + lo.c) * iz;
    double corr = mid.xy;
    if(three_d) {
      corr += (hi.xx - 2.0 * mid.xx + lo.xx) * iz;
      corr += (hi.yy - 2.0 * mid.yy + lo.yy) * iz;
      corr -= a.alpha * ((hi.xy - 2.0 * mid.xy + lo.xy) * iz);
    }
    double r = mid.c;
    r += s_gp * gp;
    r += s_dif * lap;
    r += s_adv * adv;
    if(a.has_prev) r += s_prev * prev;
    r += s_corr * corr;
    a.rhs[C][q] = r;
    lo = mid;
    mid = hi;
  }
}

// Four blocks per SM without unrolling: 445 us at 256^3 (three 611, three
// unrolled by two 574, five 505).
__global__ void __launch_bounds__(kTX* kTY, 4) k_predictor_rest(PredictorArgs a, int kchunk) {
  const Tile3 t = component_tile();
  if(t.comp == 0) predictor_tile<0>(a, t.bx, kchunk);
  else if(t.comp == 1) predictor_tile<1>(a, t.bx, kchunk);
  else predictor_tile<2>(a, t.bx, kchunk);
}

// initialize_exact_state (solver/taylor_green.cpp:335-395), active entries.
__global__ void k_tg_init(Grid g, int mode, int loc, double* f) {
  const Lay L = make_lay(g, loc);
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if(i > L.nx || j > L.ny || k > L.nz) return;
  const bool three_d = g.nz > 1;
  // coordinate_for_storage_index (core/field_layout.hpp:226-238)
  const double x = (loc == kFaceX) ? (i - 1) * g.dx : (i - 1 + 0.5) * g.dx;
  const double y = (loc == kFaceY) ? (j - 1) * g.dy : (j - 1 + 0.5) * g.dy;
  const double z = (loc == kFaceZ) ? (k - 1) * g.dz : (k - 1 + 0.5) * g.dz;
  double val = 0.0;
  if(loc == kFaceX) {
    const double zf = three_d ? cos(z) : 1.0;
    val = mode == 0 ? -cos(x) * sin(y) * zf : sin(x) * cos(y) * zf;
  } else if(loc == kFaceY) {
    const double zf = three_d ? cos(z) : 1.0;
    val = mode == 0 ? sin(x) * cos(y) * zf : -cos(x) * sin(y) * zf;
  } else if(loc == kCell) {
    const double sign = mode == 0 ? 1.0 : -1.0;
    val = three_d ? sign * -0.0625 * (cos(2.0 * x) + cos(2.0 * y)) * (cos(2.0 * z) + 2.0)
                  : sign * -0.25 * (cos(2.0 * x) + cos(2.0 * y));
  }
  f[L.idx(i, j, k)] = val;
}

}  // namespace

void launch_predictor_rhs(const PredictorArgs& a, cudaStream_t s) {
  const Launch3 l = launch3_advection(a.g);
  {
    ProfScope ps(kKAdvection, s);
    k_advect_bf<<<l.grid, l.block, 0, s>>>(a.g, a.cur[0], a.cur[1], a.cur[2], a.adv[0], a.adv[1], a.adv[2],
                                           l.kchunk);
    OFB_LAUNCH_CHECK("k_advect_bf");
  }
  launch_predictor_rest(a, s);
}

void launch_predictor_rest(const PredictorArgs& a, cudaStream_t s) {
  const Launch3 l = launch3_components(a.g);
  ProfScope ps(kKPredictor, s);
  k_predictor_rest<<<l.grid, l.block, 0, s>>>(a, l.kchunk);
  OFB_LAUNCH_CHECK("k_predictor_rest");
}

void launch_advection(const Grid& g, const double* u, const double* v, const double* w,
                      double* au, double* av, double* aw, cudaStream_t s) {
  const Launch3 l = launch3_advection(g);
  ProfScope ps(kKOther, s);
  k_advect_bf<<<l.grid, l.block, 0, s>>>(g, u, v, w, au, av, aw, l.kchunk);
  OFB_LAUNCH_CHECK("k_advection");
}

void launch_tg_init(const Grid& g, int mode, double* u, double* v, double* w, double* p,
                    cudaStream_t s) {
  double* f[4] = {p, u, v, w};
  for(int loc = 0; loc < 4; ++loc) {
    if(loc == kFaceZ) continue;  // w = 0 (solver/taylor_green.cpp:368)
    const Lay L = make_lay(g, loc);
    dim3 block(32, 8, 1);
    dim3 grid((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz);
    ProfScope ps(kKOther, s);
    k_tg_init<<<grid, block, 0, s>>>(g, mode, loc, f[loc]);
    OFB_LAUNCH_CHECK("k_tg_init");
  }
}

}  // namespace ofb
