// Projection-side kernels (solver/projection.cpp:1049-1131): divergence to
// pressure right-hand side, the Poisson system right-hand side with its
// boundary source, and one pass that corrects the velocity,
// u = u* - (dt/rho) grad(phi), with the pressure-correction ghost rules folded
// in, produces every step diagnostic and updates the total pressure.
#include "kernels.hpp"

namespace ofb {

namespace {

#define CELL_PROLOGUE(g)                                   \
  const int i = blockIdx.x * kTX + threadIdx.x;            \
  const int j = blockIdx.y * kTY + threadIdx.y;            \
  const bool valid = i < (g).nx && j < (g).ny;             \
  const int k0 = blockIdx.z * kchunk;                      \
  const int k1 = min(k0 + kchunk, (g).nz);

// build_boundary_source (linsolve/poisson_solver.cpp:635-642): the operator
// applied to a zero field with the actual boundary values.
__device__ __forceinline__ double boundary_source(const Grid& g, const PBC& pbc, int i, int j,
                                                  int k) {
  const int pos[3] = {i, j, k};
  double acc = 0.0;
#pragma unroll
  for(int a = 0; a < 3; ++a) {
    double nb = 0.0;
    const double h = g.h(a);
    const int n = g.n(a);
#pragma unroll
    for(int s = 0; s < 2; ++s) {
      const bool upper = s == 1;
      if((!upper && pos[a] > 0) || (upper && pos[a] < n - 1)) continue;
      const int type = pbc.type[2 * a + s];
      if(type == kPNeumann) nb += upper ? 0.0 + pbc.gradient[2 * a + s] * h : 0.0 - pbc.gradient[2 * a + s] * h;
      else if(type == kPDirichlet) nb += 2.0 * pbc.value[2 * a + s] - 0.0;
    }
    acc -= nb / (h * h);
  }
  return acc;
}

template <bool SOURCE>
__global__ void __launch_bounds__(kTX* kTY)
    k_divergence_rhs(Grid g, PBC pbc, const double* __restrict__ u, const double* __restrict__ v,
                     const double* __restrict__ w, double scale, double* __restrict__ rhs,
                     double* __restrict__ b, SolveScalars* sc, int zm, int kchunk, RedBuf rb) {
  CELL_PROLOGUE(g)
  const Lay P = make_lay(g, kCell), U = make_lay(g, kFaceX), V = make_lay(g, kFaceY),
            W = make_lay(g, kFaceZ);
  const CLay C = make_clay(g.nx, g.ny, g.nz);
  const double idx = 1.0 / g.dx, idy = 1.0 / g.dy, idz = 1.0 / g.dz;
  double acc[3] = {0.0, 0.0, 0.0};
  if(valid) {
    double w0 = w[W.idx(i + 1, j + 1, k0 + 1)];  // the cell's lower z face
#pragma unroll 2
    for(int k = k0; k < k1; ++k) {
      const int uq = U.idx(i + 1, j + 1, k + 1), vq = V.idx(i + 1, j + 1, k + 1);
      const double w1 = w[W.idx(i + 1, j + 1, k + 2)];
      // compute_divergence (operators/discrete_operators.cpp:98-113)
      const double div = (u[uq + 1] - u[uq]) * idx + (v[vq + V.sx] - v[vq]) * idy + (w1 - w0) * idz;
      w0 = w1;
      const double r = div * scale;
      rhs[P.idx(i + 1, j + 1, k + 1)] = r;
      double bv = -r;
      if constexpr(SOURCE) bv -= boundary_source(g, pbc, i, j, k);
      b[C.idx(i, j, k)] = bv;
      acc[0] += div * div;
      acc[1] += r * r;
      acc[2] += bv;
    }
  }
  const bool mx[3] = {false, false, false};
  const int n = C.count();
  reduce_finish<3>(acc, mx, rb, [=](const Sums<3>& s) {
    sc->div_before_l2 = sqrt(s.v[0] / n);
    sc->rhs_l2 = sqrt(s.v[1] / n);
    sc->sb = zm ? s.v[2] / n : 0.0;
    sc->removed_rhs_mean = sc->sb;
  });
}

__global__ void __launch_bounds__(kTX* kTY)
    k_rhs_to_system(Grid g, PBC pbc, const double* __restrict__ rhs, double* __restrict__ b,
                    SolveScalars* sc, int zm, int kchunk, RedBuf rb) {
  CELL_PROLOGUE(g)
  const Lay P = make_lay(g, kCell);
  const CLay C = make_clay(g.nx, g.ny, g.nz);
  double acc[1] = {0.0};
  if(valid) {
    for(int k = k0; k < k1; ++k) {
      const double bv = -rhs[P.idx(i + 1, j + 1, k + 1)] - boundary_source(g, pbc, i, j, k);
      b[C.idx(i, j, k)] = bv;
      acc[0] += bv;
    }
  }
  const bool mx[1] = {false};
  const int n = C.count();
  reduce_finish<1>(acc, mx, rb, [=](const Sums<1>& s) {
    sc->sb = zm ? s.v[0] / n : 0.0;
    sc->removed_rhs_mean = sc->sb;
  });
}

__global__ void __launch_bounds__(kTX* kTY)
    k_pressure_to_compact(Grid g, const double* __restrict__ p, double* __restrict__ x,
                          SolveScalars* sc, int zm, int kchunk, RedBuf rb) {
  CELL_PROLOGUE(g)
  const Lay P = make_lay(g, kCell);
  const CLay C = make_clay(g.nx, g.ny, g.nz);
  double acc[1] = {0.0};
  if(valid) {
    for(int k = k0; k < k1; ++k) {
      const double v = p[P.idx(i + 1, j + 1, k + 1)];
      x[C.idx(i, j, k)] = v;
      acc[0] += v;
    }
  }
  const bool mx[1] = {false};
  const int n = C.count();
  reduce_finish<1>(acc, mx, rb, [=](const Sums<1>& s) { sc->sx = zm ? s.v[0] / n : 0.0; });
}

// correct_velocity (solver/projection.cpp:1066-1095) on the active faces, the
// max |corrected - previous| reduction and the post-correction cell quantities
// -- divergence after, pressure mean, padded pressure correction, total-pressure
// update, CFL -- in one pass over the cells: a thread owns a cell's lower
// faces (and the upper one at the end of an axis), forms the upper ones again
// for the divergence and carries the z face and the next plane's pressure along
// k.  Thirteen vectors pass where the three face kernels and the cell pass moved
// nineteen (256^3: 490 + 260 us, now 345; at three blocks per SM, two take 406).
//
// The pressure-correction ghosts follow apply_pressure_boundary_conditions
// (solver/projection.cpp:302-337, 973-984): periodic image, Neumann active
// -/+ gradient h, Dirichlet 2 value - active.  The divergence and the CFL number
// use the faces as the velocity boundary conditions leave them: they already
// hold wall values and equal periodic duplicates; a fixed-pressure face takes
// its inner neighbour's value (:431-437).
__global__ void __launch_bounds__(kTX* kTY, 3)
    k_finish(FinishArgs a, SolveScalars* sc, int kchunk, RedBuf rb) {
  const Grid& g = a.g;
  CELL_PROLOGUE(g)
  const Lay P = make_lay(g, kCell);
  const Lay FL[3] = {make_lay(g, kFaceX), make_lay(g, kFaceY), make_lay(g, kFaceZ)};
  const CLay C = make_clay(g.nx, g.ny, g.nz);
  const double ih[3] = {1.0 / g.dx, 1.0 / g.dy, 1.0 / g.dz};
  const double sx = sc->sx;
  const bool update = a.p_total != nullptr && (!a.guard || sc->converged);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};  // div^2, phi, max CFL, max |dv|
  if(valid) {
    const double* __restrict__ x = a.x;
    // ghost of the cell value c across face f of axis d
    auto ghost = [&](int f, int d, double c, double wrapped) {
      const int type = a.pbc.type[f];
      if(type == kPPeriodic) return wrapped;
      if(type == kPDirichlet) return 2.0 * a.pbc.value[f] - c;
      const double step = a.pbc.gradient[f] * g.h(d);
      return (f & 1) ? c + step : c - step;
    };
    const bool xf = i == 0, xe = i == g.nx - 1, yf = j == 0, ye = j == g.ny - 1;
    const int dxl = xf ? g.nx - 1 : -1, dxh = xe ? 1 - g.nx : 1;
    const int dyl = (yf ? g.ny - 1 : -1) * g.nx, dyh = (ye ? 1 - g.ny : 1) * g.nx;
    const bool track = a.prev[0] != nullptr;
    int q = C.idx(i, j, k0);
    double c = x[q] - sx;
    const double below = k0 > 0 ? x[q - C.nxy] - sx : ghost(4, 2, c, x[q + (g.nz - 1) * C.nxy] - sx);
    int uq = FL[0].idx(i + 1, j + 1, k0 + 1), vq = FL[1].idx(i + 1, j + 1, k0 + 1),
        wq = FL[2].idx(i + 1, j + 1, k0 + 1), pq = P.idx(i + 1, j + 1, k0 + 1);
    double w0 = a.pred[2][wq] + a.scale * ((c - below) * ih[2]);  // the cell's lower z face
    for(int k = k0; k < k1; ++k) {
      const bool top = k + 1 == g.nz;
      // every load of the cell before its first store, through the read-only
      // path: the compiler may not move an ordinary load over the stores
      const double xa = __ldg(&x[top ? C.idx(i, j, 0) : q + C.nxy]);
      const double xl = __ldg(&x[q + dxl]), xh = __ldg(&x[q + dxh]), yl = __ldg(&x[q + dyl]), yh = __ldg(&x[q + dyh]);
      const double pu0 = __ldg(&a.pred[0][uq]), pu1 = __ldg(&a.pred[0][uq + 1]);
      const double pv0 = __ldg(&a.pred[1][vq]), pv1 = __ldg(&a.pred[1][vq + FL[1].sx]);
      const double pw1 = __ldg(&a.pred[2][wq + FL[2].sxy]);
      double ou = 0.0, ov = 0.0, ow = 0.0, pt = 0.0, rh = 0.0;
      if(track) {
        ou = __ldg(&a.prev[0][uq]);
        ov = __ldg(&a.prev[1][vq]);
        ow = __ldg(&a.prev[2][wq]);
      }
      if(update) {
        pt = a.p_total[pq];
        rh = __ldg(&a.rhs_padded[pq]);
      }
      const double above = top ? ghost(5, 2, c, xa - sx) : xa - sx;
      const double pl = xf ? ghost(0, 0, c, xl - sx) : xl - sx, ph = xe ? ghost(1, 0, c, xh - sx) : xh - sx;
      const double ql = yf ? ghost(2, 1, c, yl - sx) : yl - sx, qh = ye ? ghost(3, 1, c, yh - sx) : yh - sx;
      double u0 = pu0 + a.scale * ((c - pl) * ih[0]), u1 = pu1 + a.scale * ((ph - c) * ih[0]);
      double v0 = pv0 + a.scale * ((c - ql) * ih[1]), v1 = pv1 + a.scale * ((qh - c) * ih[1]);
      double w1 = pw1 + a.scale * ((above - c) * ih[2]);
      a.out[0][uq] = u0;
      a.out[1][vq] = v0;
      a.out[2][wq] = w0;
      if(xe) a.out[0][uq + 1] = u1;
      if(ye) a.out[1][vq + FL[1].sx] = v1;
      if(top) a.out[2][wq + FL[2].sxy] = w1;
      if(track) {
        acc[3] = fmax(acc[3], fmax(fabs(u0 - ou), fmax(fabs(v0 - ov), fabs(w0 - ow))));
        if(xe) acc[3] = fmax(acc[3], fabs(u1 - a.prev[0][uq + 1]));
        if(ye) acc[3] = fmax(acc[3], fabs(v1 - a.prev[1][vq + FL[1].sx]));
        if(top) acc[3] = fmax(acc[3], fabs(w1 - a.prev[2][wq + FL[2].sxy]));
      }
      const double next = w1;
      if(xf && a.open[0]) u0 = u1;
      if(xe && a.open[1]) u1 = u0;
      if(yf && a.open[2]) v0 = v1;
      if(ye && a.open[3]) v1 = v0;
      if(k == 0 && a.open[4]) w0 = w1;
      if(top && a.open[5]) w1 = w0;
      const double div = (u1 - u0) * ih[0] + (v1 - v0) * ih[1] + (w1 - w0) * ih[2];
      acc[0] += div * div;
      acc[1] += c;
      if(a.phi_padded != nullptr) a.phi_padded[pq] = c;
      if(update) {
        // p_total += phi; p_total += (-0.5 nu dt) rhs (solver/taylor_green.cpp:607-608)
        pt += c;
        pt += a.p_rhs_scale * rh;
        a.p_total[pq] = pt;
      }
      if(a.dt > 0.0) {
        // compute_advective_cfl (solver/momentum_terms.cpp:327-355)
        const double local = a.dt * (fabs(0.5 * (u0 + u1)) * ih[0] + fabs(0.5 * (v0 + v1)) * ih[1] +
                                     fabs(0.5 * (w0 + w1)) * ih[2]);
        acc[2] = fmax(acc[2], local);
      }
      w0 = next;
      c = above;
      q += C.nxy;
      uq += FL[0].sxy;
      vq += FL[1].sxy;
      wq += FL[2].sxy;
      pq += P.sxy;
    }
  }
  const bool mx[4] = {false, false, true, true};
  const int n = C.count();
  reduce_finish<4>(acc, mx, rb, [=](const Sums<4>& s) {
    sc->div_after_l2 = sqrt(s.v[0] / n);
    sc->pressure_mean = s.v[1] / n;
    sc->max_cfl = s.v[2];
    sc->max_dv = s.v[3];
    sc->nonfinite = isfinite(sc->max_dv) && isfinite(sc->div_after_l2) ? 0 : 1;
  });
}

}  // namespace

void launch_divergence_rhs(const Grid& g, const PBC& pbc, const double* u, const double* v,
                           const double* w, double scale, double* rhs_padded, double* b,
                           SolveScalars* sc, RedBuf rb, cudaStream_t s) {
  int zm = 1, with_source = 0;
  for(int f = 0; f < 6; ++f) {
    if(pbc.type[f] == kPDirichlet) zm = 0;
    if((pbc.type[f] == kPDirichlet && pbc.value[f] != 0.0) ||
       (pbc.type[f] == kPNeumann && pbc.gradient[f] != 0.0))
      with_source = 1;
  }
  const Launch3 l = launch3(g.nx, g.ny, g.nz, kReducingBlocks);
  ProfScope ps(kKDivergence, s);
  const auto kern = with_source ? k_divergence_rhs<true> : k_divergence_rhs<false>;
  kern<<<l.grid, l.block, 0, s>>>(g, pbc, u, v, w, scale, rhs_padded, b, sc, zm, l.kchunk, rb);
  OFB_LAUNCH_CHECK("k_divergence_rhs");
}

void launch_rhs_to_system(const Grid& g, const PBC& pbc, const double* rhs_padded, double* b,
                          SolveScalars* sc, RedBuf rb, cudaStream_t s) {
  int zm = 1;
  for(int f = 0; f < 6; ++f)
    if(pbc.type[f] == kPDirichlet) zm = 0;
  const Launch3 l = launch3(g.nx, g.ny, g.nz, kReducingBlocks);
  ProfScope ps(kKOther, s);
  k_rhs_to_system<<<l.grid, l.block, 0, s>>>(g, pbc, rhs_padded, b, sc, zm, l.kchunk, rb);
  OFB_LAUNCH_CHECK("k_rhs_to_system");
}

void launch_pressure_to_compact(const Grid& g, const double* p_padded, double* x,
                                SolveScalars* sc, int zm, RedBuf rb, cudaStream_t s) {
  const Launch3 l = launch3(g.nx, g.ny, g.nz, kReducingBlocks);
  ProfScope ps(kKOther, s);
  k_pressure_to_compact<<<l.grid, l.block, 0, s>>>(g, p_padded, x, sc, zm, l.kchunk, rb);
  OFB_LAUNCH_CHECK("k_pressure_to_compact");
}

void launch_finish(const FinishArgs& a, SolveScalars* sc, RedBuf rb, cudaStream_t s) {
  const Launch3 l = launch3(a.g.nx, a.g.ny, a.g.nz, kReducingBlocks);
  ProfScope ps(kKCorrect, s);
  k_finish<<<l.grid, l.block, 0, s>>>(a, sc, l.kchunk, rb);
  OFB_LAUNCH_CHECK("k_finish");
}

}  // namespace ofb
