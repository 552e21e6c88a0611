// ADI predictor sweeps (solve_component_sweep / solve_component_sweep_periodic,
// solver/projection.cpp:619-866).  Every line of one (component, axis) sweep
// has the same constant-coefficient tridiagonal matrix -- Toeplitz with
// Dirichlet/ghost-relation end rows on walls, cyclic with Sherman-Morrison on
// periodic axes -- so the Thomas factors (modified upper diagonal and inverse
// pivots) and the Sherman-Morrison correction vector are computed once on the
// host in FP64 and shared.  Lines with a moderate coupling (every projection step
// here: alpha / h^2 is well below one) are solved in chunks by sums with constant
// weights (k_adi_lines, k_adi_rows); the others by one warp per line (k_adi_scan)
// or one thread per line (k_adi_tile).
#include "kernels.hpp"

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

namespace ofb {

struct AdiAxis {
  bool active = false;      // sweep runs (n > 0)
  bool periodic = false;
  bool copy_duplicate = false;
  int n = 0;                // unknowns per line
  int begin = 0;            // storage index of the first unknown
  int dup_index = 0;        // storage index of the duplicated periodic face
  int lines = 0;
  double lower = 0.0;       // sub-diagonal (rows 1..n-1)
  double rhs_first = 0.0;   // constants added to rhs[0], rhs[n-1] on walls
  double rhs_last = 0.0;
  double uc_over_gamma = 0.0;
  double inv_den = 0.0;
  size_t off = 0;           // offset of cu/ip/z in the coefficient buffer
  // chunked solver (see solve_chunk)
  bool chunked = false;
  double lambda = 0.0, scale = 0.0, scale_lo = 0.0, fold = 0.0;  // scale + scale_lo: unevaluated
  double step = 0.0, last = 0.0, all = 0.0;  // lambda to the power of a chunk, of the last one, of the line
  double c_lo = 0.0, f_lo = 0.0, c_hi = 0.0, f_hi = 0.0, close = 0.0;  // sums beyond the ends
  // partition (warp-scan) solver, used when 64 <= n <= 1024 (n a multiple of
  // 32 on periodic axes; wall lines are padded to a multiple of 32):
  // per-lane segment factors, spikes and the interface operator, all laid
  // out [element][lane] so that a warp reads them with one coalesced load
  bool partition = false;
  int seg = 0;              // K = ceil(n / 32)
  size_t poff = 0;          // offset: cu[K][32], ip[K][32], v[K][32], w[K][32], gl[64][32], gr[64][32]
};

struct AdiPlan {
  Grid g;
  AdiAxis ax[3][3];  // [component][axis]
  double* coef = nullptr;  // device: per (comp, axis): cu[n], ip[n], z[n]
};

namespace {

// When a line takes the chunked solver.  The rounding of lambda moves the matrix
// by (1 + lambda) / (1 - lambda) rounding errors, 3.3 at alpha / h^2 = 2.5 and
// growing with its root: up to there the error against 64-bit exact solutions is
// below the eliminations' (mean over lines of 8 to 1024 unknowns and alpha / h^2
// from 1e-5 to 2.4: 2.7e-16 of the largest value, the eliminations 3.1e-16).
// Shorter lines than 8 unknowns go to k_adi_tile; a line must fit a block's threads
// (and a row its shared memory).
constexpr double kChunkMaxBeta = 2.5;
constexpr int kLineChunk = 16, kLineThreads = 1024;
constexpr int kChunkMinLine = 8, kRowMaxLine = 4096, kLineMaxLine = kLineChunk * kLineThreads;

double tangential_coef(int type) {
  return (type == kNoSlip || type == kPrescribed) ? -1.0 : (type == kSymmetry || type == kFixedPressure) ? 1.0 : 0.0;
}

void adi_attributes();

// The chunked solver's constants for the line (component c, axis a), in extended
// precision from the matrix that the eliminations take -- its diagonal is 1 + 2
// beta as rounded -- and from the rounded lambda: the weights of the solution then
// add up to one over the row's sum, the factor that carries that kept to twice the
// precision (its rounding would act the same way in every sweep).  Appends lambda^(distance to either end) of the chunks
// to `host`.
void chunked_line(AdiAxis& A, double beta, const VBC& bc, int c, int a, std::vector<double>& host) {
  using R = long double;
  const int n = A.n, S = kLineChunk, chunks = (n + S - 1) / S;
  A.chunked = true;
  const double diagonal = 1.0 + 2.0 * beta;
  const R row = diagonal - 2.0L * beta;  // 1 but for that rounding
  A.lambda = static_cast<double>(2.0L * beta / (diagonal + std::sqrt(row * (diagonal + 2.0L * beta))));
  const R l = A.lambda;
  auto power = [&](int k) { return static_cast<double>(std::pow(l, static_cast<R>(k))); };
  const R scale = (1.0L - l) * (1.0L - l) / row;
  // rounded down: the rest is positive, and an infinity is not multiplied into a NaN
  A.scale = std::nextafter(static_cast<double>(scale), 0.0);
  A.scale_lo = static_cast<double>(scale - A.scale);
  A.fold = static_cast<double>(1.0L / (1.0L - l * l));
  A.step = power(S);
  A.last = power(n - S * (chunks - 1));
  A.all = power(n);
  // what lies beyond a wall: r there is the image add + sign r, or at a node
  // the wall's value and the image about it
  const R about_node = row * (1.0L + l) / (1.0L - l), about_face = row * 2.0L / (1.0L - l);
  auto wall = [&](int face, double& constant, double& factor) {
    const int type = bc.type[face];
    const bool node = c == a && is_dirichlet_velocity(type);
    const bool fixed = node || type == kNoSlip || type == kPrescribed;
    constant = fixed ? static_cast<double>(bc.vel[face][c] * (node ? about_node : about_face)) : 0.0;
    factor = node ? -A.lambda : fixed ? -1.0 : 1.0;
  };
  if(A.periodic) {
    A.close = static_cast<double>(1.0L / (1.0L - std::pow(l, static_cast<R>(n))));
  } else {
    wall(2 * a, A.c_lo, A.f_lo);
    wall(2 * a + 1, A.c_hi, A.f_hi);
    A.close = static_cast<double>(1.0L / (1.0L - R(A.f_lo) * A.f_hi * std::pow(l, static_cast<R>(2 * n))));
  }
  for(int q = 0; q < chunks; ++q) host.push_back(power(q * S));
  for(int q = 0; q < chunks; ++q) host.push_back(power(n - std::min(n, (q + 1) * S)));
}

}  // namespace

AdiPlan* adi_plan_create(const Grid& g, const VBC& bc, double alpha) {
  std::unique_ptr<AdiPlan, void (*)(AdiPlan*)> plan(new AdiPlan(), adi_plan_destroy);
  AdiPlan* const p = plan.get();
  p->g = g;
  std::vector<double> host;
  for(int c = 0; c < 3; ++c) {
    const Lay L = make_lay(g, kFaceX + c);
    for(int a = 0; a < 3; ++a) {
      AdiAxis& A = p->ax[c][a];
      const double h = g.h(a);
      const double beta = alpha / (h * h);
      const bool periodic = bc.type[2 * a] == kPeriodic;
      int begin = 1, end = 1 + L.n(a);
      if(periodic) {
        if(c == a) end -= 1;
      } else if(c == a) {
        begin += is_dirichlet_velocity(bc.type[2 * a]) ? 1 : 0;
        end -= is_dirichlet_velocity(bc.type[2 * a + 1]) ? 1 : 0;
      }
      const int n = end - begin;
      int a1 = a == 0 ? 1 : 0, a2 = a == 2 ? 1 : 2;
      A.lines = L.n(a1) * L.n(a2);
      if(n <= 0) continue;
      A.active = true;
      A.periodic = periodic;
      A.n = n;
      A.begin = begin;
      A.copy_duplicate = periodic && c == a;
      A.dup_index = L.n(a);  // active_end - 1
      A.lower = -beta;
      A.off = host.size();
      if(beta > 0.0 && beta <= kChunkMaxBeta && n >= kChunkMinLine && n <= (a == 0 ? kRowMaxLine : kLineMaxLine)) {
        chunked_line(A, beta, bc, c, a, host);
        continue;
      }
      std::vector<double> di(n, 1.0 + 2.0 * beta), up(n, -beta), lo(n, -beta);
      lo[0] = 0.0;
      up[n - 1] = 0.0;
      std::vector<double> cu(n), ip(n), z(n, 0.0);
      if(periodic) {
        const double lc = -beta, uc = -beta;
        if(n == 1) {
          // solve_cyclic_tridiagonal n == 1 (solver/projection.cpp:574-581)
          const double pivot = di[0] + lc + uc;
          if(std::fabs(pivot) < 1.0e-30) {
            throw std::runtime_error("cyclic tridiagonal solve encountered a zero pivot");
          }
          cu[0] = 0.0;
          ip[0] = 1.0 / pivot;
          A.uc_over_gamma = 0.0;
          A.inv_den = 0.0;
        } else {
          const double gamma = -di[0];
          std::vector<double> dm = di;
          dm[0] = di[0] - gamma;
          dm[n - 1] = di[n - 1] - lc * uc / gamma;
          // Thomas factors of the modified matrix
          double pivot = dm[0];
          cu[0] = n > 1 ? up[0] / pivot : 0.0;
          ip[0] = 1.0 / pivot;
          for(int q = 1; q < n; ++q) {
            pivot = dm[q] - lo[q] * cu[q - 1];
            if(std::fabs(pivot) < 1.0e-30) {
              throw std::runtime_error("tridiagonal solve encountered a zero pivot");
            }
            cu[q] = q + 1 < n ? up[q] / pivot : 0.0;
            ip[q] = 1.0 / pivot;
          }
          // z = M^-1 u with u = (gamma, 0, ..., 0, lower_corner), as the
          // reference's second Thomas solve (solver/projection.cpp:600-605)
          std::vector<double> mr(n), uvec(n, 0.0);
          uvec[0] = gamma;
          uvec[n - 1] = lc;
          double pv = dm[0];
          std::vector<double> mu(n);
          mu[0] = up[0] / pv;
          mr[0] = uvec[0] / pv;
          for(int q = 1; q < n; ++q) {
            pv = dm[q] - lo[q] * mu[q - 1];
            mu[q] = q + 1 < n ? up[q] / pv : 0.0;
            mr[q] = (uvec[q] - lo[q] * mr[q - 1]) / pv;
          }
          z[n - 1] = mr[n - 1];
          for(int q = n - 1; q-- > 0;) z[q] = mr[q] - mu[q] * z[q + 1];
          const double den = 1.0 + z[0] + uc * z[n - 1] / gamma;
          if(std::fabs(den) < 1.0e-30) {
            throw std::runtime_error(
                "cyclic tridiagonal solve encountered a singular Sherman-Morrison update");
          }
          A.uc_over_gamma = uc / gamma;
          A.inv_den = 1.0 / den;
        }
      } else {
        // wall rows (solver/projection.cpp:757-780)
        const int lo_t = bc.type[2 * a], hi_t = bc.type[2 * a + 1];
        double r0 = 0.0, rn = 0.0;
        if(c == a && is_dirichlet_velocity(lo_t)) {
          r0 += beta * bc.vel[2 * a][a];
        } else {
          di[0] -= beta * tangential_coef(lo_t);
          r0 += beta * ((lo_t == kNoSlip || lo_t == kPrescribed) ? 2.0 * bc.vel[2 * a][c] : 0.0);
        }
        if(c == a && is_dirichlet_velocity(hi_t)) {
          rn += beta * bc.vel[2 * a + 1][a];
        } else {
          di[n - 1] -= beta * tangential_coef(hi_t);
          rn += beta * ((hi_t == kNoSlip || hi_t == kPrescribed) ? 2.0 * bc.vel[2 * a + 1][c] : 0.0);
        }
        A.rhs_first = r0;
        A.rhs_last = rn;
        double pivot = di[0];
        if(std::fabs(pivot) < 1.0e-30) {
          throw std::runtime_error("tridiagonal solve encountered a zero pivot");
        }
        cu[0] = n > 1 ? up[0] / pivot : 0.0;
        ip[0] = 1.0 / pivot;
        for(int q = 1; q < n; ++q) {
          pivot = di[q] - lo[q] * cu[q - 1];
          if(std::fabs(pivot) < 1.0e-30) {
            throw std::runtime_error("tridiagonal solve encountered a zero pivot");
          }
          cu[q] = q + 1 < n ? up[q] / pivot : 0.0;
          ip[q] = 1.0 / pivot;
        }
      }
      host.insert(host.end(), cu.begin(), cu.end());
      host.insert(host.end(), ip.begin(), ip.end());
      host.insert(host.end(), z.begin(), z.end());
      if(n >= 64 && (n + 31) / 32 <= 32 && (n % 32 == 0 || !periodic)) {
        // Warp-scan form of the two Thomas recurrences (lane p owns the
        // unknowns q = pK + j, j < K):
        //   forward  m_q = ip_q r_q + f_q m_{q-1},  f_q = -lower ip_q
        //   backward x_q = m_q + g_q x_{q+1},       g_q = -cu_q
        // Lane-local products of f (resp. g) and the per-step multipliers of
        // the Kogge-Stone scans are line-independent and stored here.  A line
        // whose n is not a multiple of 32 (walls) is padded to 32 K unknowns
        // with ip = cu = 0: the padding decouples (m = x = 0 there) and the
        // real unknowns are unchanged.  Periodic lines are not padded (the
        // Sherman-Morrison update reads the last unknown from lane 31).
        const int P = 32, K = (n + 31) / 32;
        std::vector<double> fB(K * P), gD(K * P), ipj(K * P), cuj(K * P), zj(K * P);
        std::vector<double> mf(5 * P, 0.0), mb(5 * P, 0.0);
        std::vector<double> lane_f(P), lane_g(P);
        for(int lane = 0; lane < P; ++lane) {
          double prod = 1.0;
          for(int j = 0; j < K; ++j) {
            const int q = lane * K + j;
            const double ipq = q < n ? ip[q] : 0.0;
            const double f = q == 0 ? 0.0 : -(-beta) * ipq;
            prod = j == 0 ? f : prod * f;
            fB[j * P + lane] = prod;
            ipj[j * P + lane] = ipq;
            cuj[j * P + lane] = q < n ? cu[q] : 0.0;
            zj[j * P + lane] = q < n ? z[q] : 0.0;
          }
          lane_f[lane] = prod;  // m_end = A + prod * m_in
          double dprod = 1.0;
          for(int j = K - 1; j >= 0; --j) {
            const int q = lane * K + j;
            const double g = q < n ? -cu[q] : 0.0;
            dprod = j == K - 1 ? g : dprod * g;
            gD[j * P + lane] = dprod;
          }
          lane_g[lane] = dprod;  // x_first = C + dprod * x_in
        }
        // Kogge-Stone multipliers: inclusive scan of (a, b) maps; step s
        // combines lane p with lane p - 2^s (forward) / p + 2^s (backward)
        std::vector<double> cf = lane_f, cb = lane_g;
        for(int st = 0; st < 5; ++st) {
          const int d = 1 << st;
          std::vector<double> nf = cf, nb = cb;
          for(int lane = 0; lane < P; ++lane) {
            mf[st * P + lane] = lane >= d ? cf[lane] : 0.0;
            if(lane >= d) nf[lane] = cf[lane] * cf[lane - d];
            mb[st * P + lane] = lane + d < P ? cb[lane] : 0.0;
            if(lane + d < P) nb[lane] = cb[lane] * cb[lane + d];
          }
          cf = nf;
          cb = nb;
        }
        A.partition = true;
        A.seg = K;
        A.poff = host.size();
        for(auto* v : {&ipj, &fB, &cuj, &gD, &zj}) host.insert(host.end(), v->begin(), v->end());
        host.insert(host.end(), mf.begin(), mf.end());
        host.insert(host.end(), mb.begin(), mb.end());
      }
    }
  }
  adi_attributes();
  if(!host.empty()) {
    OFB_CHECK(cudaMalloc(&p->coef, host.size() * sizeof(double)));
    OFB_CHECK(cudaMemcpy(p->coef, host.data(), host.size() * sizeof(double), cudaMemcpyHostToDevice));
    OFB_CHECK(cudaStreamSynchronize(nullptr));  // the context's stream does not wait for the default one
  }
  return plan.release();
}

void adi_plan_destroy(AdiPlan* p) {
  if(p == nullptr) return;
  if(p->coef) cudaFree(p->coef);
  delete p;
}

int adi_line_count(const AdiPlan* p, int comp, int axis) {
  return p->ax[comp][axis].active ? p->ax[comp][axis].lines : 0;
}

bool adi_axis_active(const AdiPlan* p, int comp, int axis) { return p->ax[comp][axis].active; }

void adi_axis_geometry(const AdiPlan* p, int comp, int axis, int* begin, int* n) {
  *begin = p->ax[comp][axis].begin;
  *n = p->ax[comp][axis].n;
}

namespace {

struct SweepArgs {
  Lay L;
  int axis;
  int n, begin, dup_index, periodic, copy_duplicate;
  double lower, rhs_first, rhs_last, uc_over_gamma, inv_den;
  const double* cu;
  const double* ip;
  const double* z;
};

// Shared-memory line solver: one warp stages `lines` whole lines in shared
// memory (coalesced: x-lines load row segments, y/z-lines load 32 adjacent
// i-lines so each warp load is one contiguous row), solves them there with
// the shared Thomas factors and the Sherman-Morrison update, and stores them
// back coalesced.  Lines of an x-sweep are stored [line][n + 1] (the pad
// spreads a warp's column accesses over the banks), lines of a y/z sweep
// [n][lines] (a warp reads one row).
template <bool XLINES>
__global__ void __launch_bounds__(32) k_adi_tile(SweepArgs a, const double* __restrict__ in,
                                                 double* __restrict__ out, int lines) {
  extern __shared__ double tile[];
  const Lay& L = a.L;
  const int axis = a.axis;
  const int a1 = axis == 0 ? 1 : 0;
  const int a2 = axis == 2 ? 1 : 2;
  const int n = a.n;
  const int st = L.stride(axis);
  const int t = threadIdx.x;
  const int n1 = L.n(a1);
  const int n2 = L.n(a2);
  // line l of this block -> storage base of its position 0 along the axis
  auto line_base = [&](int l, bool& ok) {
    int c1, c2;
    if(XLINES) {
      const int flat = blockIdx.x * lines + l;
      c1 = flat % n1;
      c2 = flat / n1;
      ok = c2 < n2;
    } else {
      c1 = blockIdx.x * lines + l;
      c2 = blockIdx.y;
      ok = c1 < n1;
    }
    if(!ok) {
      c1 = 0;
      c2 = 0;
    }
    int c[3] = {0, 0, 0};
    c[a1] = c1 + 1;
    c[a2] = c2 + 1;
    return L.idx(c[0], c[1], c[2]) + a.begin * st;
  };
  auto at = [&](int l, int q) -> double& {
    return XLINES ? tile[l * (n + 1) + q] : tile[q * lines + l];
  };
  // load
  if(XLINES) {
    for(int l = 0; l < lines; ++l) {
      bool ok;
      const int base = line_base(l, ok);
      if(!ok) continue;
      for(int q = t; q < n; q += 32) at(l, q) = in[base + q];
    }
  } else {
    for(int q = 0; q < n; ++q) {
      for(int l = t; l < lines; l += 32) {
        bool ok;
        const int base = line_base(l, ok);
        if(ok) at(l, q) = in[base + q * st];
      }
    }
  }
  __syncwarp();
  // solve line t
  if(t < lines) {
    double r = at(t, 0) + a.rhs_first;
    if(n == 1) r += a.rhs_last;
    double m = r * __ldg(&a.ip[0]);
    at(t, 0) = m;
    for(int q = 1; q < n; ++q) {
      double rq = at(t, q);
      if(q == n - 1) rq += a.rhs_last;
      m = (rq - a.lower * m) * __ldg(&a.ip[q]);
      at(t, q) = m;
    }
    const double x_last = m;
    double x = m;
    for(int q = n - 2; q >= 0; --q) {
      x = at(t, q) - __ldg(&a.cu[q]) * x;
      at(t, q) = x;
    }
    if(a.periodic && n > 1) {
      const double factor = (x + a.uc_over_gamma * x_last) * a.inv_den;
      for(int q = 0; q < n; ++q) at(t, q) -= factor * __ldg(&a.z[q]);
    }
  }
  __syncwarp();
  // store (and the duplicated periodic face)
  if(XLINES) {
    for(int l = 0; l < lines; ++l) {
      bool ok;
      const int base = line_base(l, ok);
      if(!ok) continue;
      for(int q = t; q < n; q += 32) out[base + q] = at(l, q);
      if(a.copy_duplicate && t == 0) out[base - a.begin * st + a.dup_index * st] = at(l, 0);
    }
  } else {
    for(int q = 0; q < n; ++q) {
      for(int l = t; l < lines; l += 32) {
        bool ok;
        const int base = line_base(l, ok);
        if(ok) out[base + q * st] = at(l, q);
      }
    }
    if(a.copy_duplicate) {
      for(int l = t; l < lines; l += 32) {
        bool ok;
        const int base = line_base(l, ok);
        if(ok) out[base - a.begin * st + a.dup_index * st] = at(l, 0);
      }
    }
  }
}

constexpr size_t kAdiTileBytes = 64 * 1024;

struct ScanArgs {
  const double* ip;  // [K][32]
  const double* fB;  // lane-local forward products
  const double* cu;
  const double* gD;  // lane-local backward products
  const double* z;   // Sherman-Morrison vector
  const double* mf;  // [5][32] forward scan multipliers
  const double* mb;  // [5][32] backward scan multipliers
  int K;
};

// Warp-scan line solver: a block of LB warps stages LB lines in shared
// memory (element q = pK + j of a line at [j][p], so a warp's accesses are
// conflict-free); warp w solves line w.  Lane p evaluates its K forward
// elimination steps as an affine map of the unknown carried in from lane p-1,
// the 32 maps are composed by a Kogge-Stone scan over shuffles, and the same
// is done for back substitution; the periodic Sherman-Morrison update
// (solver/projection.cpp:607-616) follows.  Same Thomas factors as the
// reference's recurrences; the association of the products differs, so
// results agree to rounding.
template <bool XLINES, int LB>
__global__ void __launch_bounds__(32 * LB) k_adi_scan(SweepArgs a, ScanArgs sa,
                                                      const double* __restrict__ in,
                                                      double* __restrict__ out) {
  extern __shared__ double tile[];
  const Lay& L = a.L;
  const int axis = a.axis;
  const int a1 = axis == 0 ? 1 : 0;
  const int a2 = axis == 2 ? 1 : 2;
  const int n = a.n;
  const int K = sa.K;
  const int S = 32 * K + 1;  // per-line stride in the tile (n padded to 32 K)
  const int st = L.stride(axis);
  const int n1 = L.n(a1), n2 = L.n(a2);
  const int tid = threadIdx.x + 32 * threadIdx.y;
  const int lane = threadIdx.x, wl = threadIdx.y;
  auto line_base = [&](int l, bool& ok) {
    int c1, c2;
    if(XLINES) {
      const int flat = blockIdx.x * LB + l;
      c1 = flat % n1;
      c2 = flat / n1;
      ok = c2 < n2;
    } else {
      c1 = blockIdx.x * LB + l;
      c2 = blockIdx.y;
      ok = c1 < n1;
    }
    if(!ok) c1 = c2 = 0;
    int c[3] = {0, 0, 0};
    c[a1] = c1 + 1;
    c[a2] = c2 + 1;
    return L.idx(c[0], c[1], c[2]) + a.begin * st;
  };
  // element q = pK + j of a line sits at row j, column (p + rot j) mod 32 of
  // the line's tile.  On x lines a warp stages consecutive q (32 / K
  // consecutive p per j): the rotation spreads those accesses over all bank
  // groups and keeps the solve's row accesses (fixed j, lanes p = 0..31) a
  // permutation.  Other lines stage 16 lines x 2 elements per warp, already
  // spread by the odd line stride, so they keep rot = 0.
  const int rot = XLINES ? (K < 32 ? 32 / K : 1) : 0;
  auto col = [&](int j, int p) { return j * 32 + ((p + rot * j) & 31); };
  auto slot = [&](int l, int q) { return l * S + col(q % K, q / K); };
  // staged lines; the padding past n is zero
  if(XLINES) {
    bool ok;
    const int base = line_base(wl, ok);
    if(ok)
      for(int q = lane; q < 32 * K; q += 32) tile[slot(wl, q)] = q < n ? in[base + q] : 0.0;
  } else {
    const int l = tid % LB;
    bool ok;
    const int base = line_base(l, ok);
    if(ok)
      for(int q = tid / LB; q < 32 * K; q += 32) tile[slot(l, q)] = q < n ? in[base + q * st] : 0.0;
  }
  __syncthreads();
  {
    double* line = tile + wl * S;
    // forward elimination, lane-local part: m_{pK+j} = A_j + fB_j m_in
    double acc = 0.0;
    for(int j = 0; j < K; ++j) {
      const int q = lane * K + j;
      double r = line[col(j, lane)];
      if(q == 0) r += a.rhs_first;
      if(q == n - 1) r += a.rhs_last;
      const double ipq = __ldg(&sa.ip[j * 32 + lane]);
      // f_q = lower_coupling * ip_q with the coupling -(-beta) folded in
      const double f = q == 0 ? 0.0 : -a.lower * ipq;
      acc = j == 0 ? r * ipq : r * ipq + f * acc;
      line[col(j, lane)] = acc;  // A_j
    }
    // inclusive scan of lane maps: val = m at the lane's last unknown
    double val = acc;
#pragma unroll
    for(int s = 0; s < 5; ++s) {
      const double up = __shfl_up_sync(0xffffffffu, val, 1 << s);
      val += __ldg(&sa.mf[s * 32 + lane]) * up;
    }
    double m_in = __shfl_up_sync(0xffffffffu, val, 1);
    if(lane == 0) m_in = 0.0;
    for(int j = 0; j < K; ++j) {
      const double v = line[col(j, lane)] + __ldg(&sa.fB[j * 32 + lane]) * m_in;
      line[col(j, lane)] = v;  // m_q
    }
    // back substitution, lane-local: x_{pK+j} = C_j + gD_j x_in
    double cacc = 0.0;
    for(int j = K - 1; j >= 0; --j) {
      const double mq = line[col(j, lane)];
      cacc = j == K - 1 ? mq : mq - __ldg(&sa.cu[j * 32 + lane]) * cacc;
      line[col(j, lane)] = cacc;  // C_j
    }
    double bval = cacc;
#pragma unroll
    for(int s = 0; s < 5; ++s) {
      const double dn = __shfl_down_sync(0xffffffffu, bval, 1 << s);
      bval += __ldg(&sa.mb[s * 32 + lane]) * dn;
    }
    double x_in = __shfl_down_sync(0xffffffffu, bval, 1);
    if(lane == 31) x_in = 0.0;
    double x0 = 0.0, xl = 0.0;
    for(int j = 0; j < K; ++j) {
      const double x = line[col(j, lane)] + __ldg(&sa.gD[j * 32 + lane]) * x_in;
      line[col(j, lane)] = x;
      if(j == 0) x0 = x;
      if(j == K - 1) xl = x;
    }
    if(a.periodic) {
      const double first = __shfl_sync(0xffffffffu, x0, 0);
      const double last = __shfl_sync(0xffffffffu, xl, 31);
      const double factor = (first + a.uc_over_gamma * last) * a.inv_den;
      for(int j = 0; j < K; ++j) line[col(j, lane)] -= factor * __ldg(&sa.z[j * 32 + lane]);
    }
  }
  __syncthreads();
  if(XLINES) {
    bool ok;
    const int base = line_base(wl, ok);
    if(ok) {
      for(int q = lane; q < n; q += 32) out[base + q] = tile[slot(wl, q)];
      if(a.copy_duplicate && lane == 0) out[base - a.begin * st + a.dup_index * st] = tile[slot(wl, 0)];
    }
  } else {
    const int l = tid % LB;
    bool ok;
    const int base = line_base(l, ok);
    if(ok) {
      for(int q = tid / LB; q < n; q += 32) out[base + q * st] = tile[slot(l, q)];
      if(a.copy_duplicate && tid < LB) out[base - a.begin * st + a.dup_index * st] = tile[slot(l, 0)];
    }
  }
}

template <int LB>
void launch_scan(const SweepArgs& a, const ScanArgs& sa, int axis, int a1, int a2, const double* in,
                 double* out, cudaStream_t s) {
  const size_t smem = static_cast<size_t>(LB) * (32 * sa.K + 1) * sizeof(double);
  const dim3 block(32, LB, 1);
  if(axis == 0) {
    const long long nl = static_cast<long long>(a.L.n(a1)) * a.L.n(a2);
    const dim3 grid(static_cast<unsigned>((nl + LB - 1) / LB), 1, 1);
    k_adi_scan<true, LB><<<grid, block, smem, s>>>(a, sa, in, out);
  } else {
    const dim3 grid((a.L.n(a1) + LB - 1) / LB, a.L.n(a2), 1);
    k_adi_scan<false, LB><<<grid, block, smem, s>>>(a, sa, in, out);
  }
}

// ---------------------------------------------------------------------------
// Chunked line solver.  (1 + 2 beta) x_q - beta (x_{q-1} + x_{q+1}) = r_q on an
// infinite line has the solution x_q = (1 - lambda) / (1 + lambda) sum over p of
// lambda^|q - p| r_p, with lambda the smaller root of beta l^2 - (1 + 2 beta) l +
// beta = 0.  A line's ends are images that r obeys as x does: periodic wrap, or
// the reflection a wall row stands for (its ghost relation x_{-1} = add + sign
// x_0, or x_{-1} = the wall's value at a node and x_{-1-q} = add - x_{-1+q}
// beyond it).  So with the sums up to each end of a chunk,
//   m_q = r_q + lambda m_{q-1}  (all r below),   b_q = r_q + lambda b_{q+1}  (all above),
// the chunk is solved by m_q and y_q = m_q + lambda y_{q+1}, x = (1 - lambda)^2 y (the
// factor as chunked_line rounds it).
// A thread holds a chunk of kLineChunk unknowns; the sums of the chunks below and
// above it, and of the images (geometric series of the line's own two sums),
// meet in shared memory.  Every term counts, however far: weights are positive, so
// a small unknown far from a large r keeps its relative accuracy.
//
// Bound: one read and one write of each field (42 us per component and sweep at
// 256^3).  Three components take 194 us; starting a chunk as many cells early as
// lambda^cells needs to vanish took 219 (2 x 7 redundant reads per 16 unknowns,
// and the terms beyond dropped), one scan per line (k_adi_scan) 366.  At 128^3
// 30 instead of 39 us, at 128^2 8.6 instead of 10.2 (sweeps of y, z and x).
// ---------------------------------------------------------------------------
struct LineArgs {
  Lay L;
  int n, begin, dup_index, periodic, copy_duplicate, chunks;
  double lambda, scale, scale_lo, fold, step, last, all;
  double c_lo, f_lo, c_hi, f_hi, close;
  const double* from_lo;  // [chunks] lambda^(unknowns below the chunk)
  const double* from_hi;  // [chunks] lambda^(unknowns above the chunk)
  const double* in;
  double* out;
};

struct Lines3 {
  LineArgs c[3];  // the components of this launch
};

// Exclusive sums over the chunks of a line, in place; the whole line's sum goes
// behind them.  Four loads at a time: a chain of single ones would wait for
// shared memory at every chunk.
__device__ __forceinline__ void sum_chunks(const LineArgs& a, double* v, int lanes, bool up) {
  double s = 0.0;
  for(int q0 = 0; q0 < a.chunks; q0 += 4) {
    double t[4];
#pragma unroll
    for(int u = 0; u < 4; ++u) t[u] = q0 + u < a.chunks ? v[(up ? q0 + u : a.chunks - 1 - q0 - u) * lanes] : 0.0;
#pragma unroll
    for(int u = 0; u < 4; ++u) {
      if(q0 + u >= a.chunks) break;
      const int q = up ? q0 + u : a.chunks - 1 - q0 - u;
      v[q * lanes] = s;
      s = (q == a.chunks - 1 ? a.last : a.step) * s + t[u];
    }
  }
  v[a.chunks * lanes] = s;
}

// r of chunk c of the block's line `lane` (zero past the line's end) to x.  F and
// B have (chunks + 1) x lanes entries.  All threads of the block call it.
__device__ __forceinline__ void solve_chunk(const LineArgs& a, double (&y)[kLineChunk], int c, int lane, int lanes,
                                            double* F, double* B) {
  constexpr int S = kLineChunk;
  const bool own = c < a.chunks;
  const int count = own ? min(S, a.n - c * S) : 0;
  const double l = a.lambda;
  double m = 0.0, b = 0.0;
#pragma unroll
  for(int t = 0; t < S; ++t)
    if(t < count) m = l * m + y[t];
#pragma unroll
  for(int t = S - 1; t >= 0; --t) b = l * b + y[t];
  if(own) {
    F[c * lanes + lane] = m;
    B[c * lanes + lane] = b;
  }
  __syncthreads();
  if(c == 0) sum_chunks(a, F + lane, lanes, true);
  if(c == (a.chunks > 1 ? 1 : 0)) sum_chunks(a, B + lane, lanes, false);
  __syncthreads();
  if(!own) return;
  const double up = F[a.chunks * lanes + lane], down = B[a.chunks * lanes + lane];
  double below, above;  // sums of the images beyond the line's ends
  if(a.periodic) {
    below = up * a.close;
    above = down * a.close;
  } else {
    below = (a.c_lo + a.f_lo * (down + a.all * (a.c_hi + a.f_hi * up))) * a.close;
    above = a.c_hi + a.f_hi * (up + a.all * below);
  }
  m = F[c * lanes + lane] + a.from_lo[c] * below;
  b = B[c * lanes + lane] + a.from_hi[c] * above;
#pragma unroll
  for(int t = 0; t < S; ++t)
    if(t < count) {
      m = l * m + y[t];
      y[t] = m;
    }
  double v = (l * m + b) * a.fold;
#pragma unroll
  for(int t = S - 1; t >= 0; --t)
    if(t < count) {
      v = l * v + y[t];
      y[t] = a.scale * v + a.scale_lo * v;
    }
}

// y and z sweeps: a block solves `lanes` lines adjacent in x (coalesced rows), a
// thread one chunk of one of them; reads and writes the field once.
__global__ void __launch_bounds__(kLineThreads, 1) k_adi_lines(Lines3 s, int axis, int lanes) {
  extern __shared__ double line_sm[];
  const LineArgs& a = s.c[blockIdx.y];
  const Lay& L = a.L;
  const int iblocks = (L.nx + lanes - 1) / lanes;
  const int other = axis == 1 ? 2 : 1;
  const int lane = threadIdx.x % lanes, c = threadIdx.x / lanes;
  const int i = (blockIdx.x % iblocks) * lanes + lane, o = blockIdx.x / iblocks;
  if(o >= L.n(other)) return;
  const int q0 = c * kLineChunk;
  const bool work = i < L.nx && c < a.chunks;
  const int st = L.stride(axis);
  const int at = L.idx(i + 1, axis == 1 ? 0 : o + 1, axis == 1 ? o + 1 : 0);
  const double* in = a.in + at + (a.begin + q0) * st;
  double y[kLineChunk];
#pragma unroll
  for(int t = 0; t < kLineChunk; ++t) y[t] = work && q0 + t < a.n ? in[t * st] : 0.0;
  solve_chunk(a, y, c, lane, lanes, line_sm, line_sm + (a.chunks + 1) * lanes);
  if(!work) return;
  double* out = a.out + at + (a.begin + q0) * st;
#pragma unroll
  for(int t = 0; t < kLineChunk; ++t)
    if(q0 + t < a.n) out[t * st] = y[t];
  if(a.copy_duplicate && q0 == 0) a.out[at + a.dup_index * st] = y[0];
}

// x sweeps: a block stages whole rows in shared memory (odd row stride: lanes
// on adjacent rows touch different banks), a thread solves one chunk of one row,
// and the rows are stored back from shared memory (coalesced both ways).
__global__ void __launch_bounds__(kLineThreads, 1) k_adi_rows(Lines3 s, int rows) {
  extern __shared__ double line_sm[];
  const LineArgs& a = s.c[blockIdx.y];
  const Lay& L = a.L;
  const int total = L.ny * L.nz;
  const int first = blockIdx.x * rows;
  if(first >= total) return;
  const int stride = a.n | 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  for(int l = warp; l < rows && first + l < total; l += warps) {
    const int at = L.idx(a.begin, (first + l) % L.ny + 1, (first + l) / L.ny + 1);
    for(int q = lane; q < a.n; q += 32) line_sm[l * stride + q] = a.in[at + q];
  }
  __syncthreads();
  const int l = threadIdx.x % rows, c = threadIdx.x / rows, q0 = c * kLineChunk;
  const bool work = c < a.chunks && first + l < total;
  double y[kLineChunk];
  double* mine = line_sm + l * stride + q0;
#pragma unroll
  for(int t = 0; t < kLineChunk; ++t) y[t] = work && q0 + t < a.n ? mine[t] : 0.0;
  double* F = line_sm + rows * stride;
  solve_chunk(a, y, c, l, rows, F, F + (a.chunks + 1) * rows);
  if(work) {
#pragma unroll
    for(int t = 0; t < kLineChunk; ++t)
      if(q0 + t < a.n) mine[t] = y[t];
  }
  __syncthreads();
  for(int w = warp; w < rows && first + w < total; w += warps) {
    const int at = L.idx(a.begin, (first + w) % L.ny + 1, (first + w) / L.ny + 1);
    for(int q = lane; q < a.n; q += 32) a.out[at + q] = line_sm[w * stride + q];
    if(a.copy_duplicate && lane == 0) a.out[at - a.begin + a.dup_index] = line_sm[w * stride];
  }
}

void launch_chunked(const AdiPlan* p, const int* comps, int count, int axis, const double* const* in,
                    double* const* out, cudaStream_t s) {
  Lines3 q{};
  int longest = 0, most_rows = 0;
  for(int t = 0; t < count; ++t) {
    const AdiAxis& A = p->ax[comps[t]][axis];
    LineArgs& a = q.c[t];
    a.L = make_lay(p->g, kFaceX + comps[t]);
    a.n = A.n;
    a.begin = A.begin;
    a.dup_index = A.dup_index;
    a.periodic = A.periodic ? 1 : 0;
    a.copy_duplicate = A.copy_duplicate ? 1 : 0;
    a.chunks = (A.n + kLineChunk - 1) / kLineChunk;
    a.lambda = A.lambda;
    a.scale = A.scale;
    a.scale_lo = A.scale_lo;
    a.fold = A.fold;
    a.step = A.step;
    a.last = A.last;
    a.all = A.all;
    a.c_lo = A.c_lo;
    a.f_lo = A.f_lo;
    a.c_hi = A.c_hi;
    a.f_hi = A.f_hi;
    a.close = A.close;
    a.from_lo = p->coef + A.off;
    a.from_hi = a.from_lo + a.chunks;
    a.in = in[comps[t]];
    a.out = out[comps[t]];
    longest = std::max(longest, A.n);
    most_rows = std::max(most_rows, a.L.ny * a.L.nz);
  }
  const int chunks = (longest + kLineChunk - 1) / kLineChunk;
  ProfScope ps(kKAdi, s);
  if(axis != 0) {
    int lanes = 32;
    while(lanes * chunks > kLineThreads) lanes /= 2;
    long long blocks = 0;
    for(int t = 0; t < count; ++t) {
      const Lay& L = q.c[t].L;
      blocks = std::max(blocks, static_cast<long long>((L.nx + lanes - 1) / lanes) * L.n(axis == 1 ? 2 : 1));
    }
    const size_t smem = 2 * static_cast<size_t>(chunks + 1) * lanes * sizeof(double);
    k_adi_lines<<<dim3(static_cast<unsigned>(blocks), count), lanes * chunks, smem, s>>>(q, axis, lanes);
    OFB_LAUNCH_CHECK("k_adi_lines");
    return;
  }
  // 16 rows per block (4 when that leaves fewer than two blocks per SM, or a
  // row so long that 16 pass the block's threads or 100 KB)
  const size_t row = (static_cast<size_t>(longest | 1) + 2 * (chunks + 1)) * sizeof(double);
  int rows = 16;
  if(most_rows < 2 * 148 * 16 || rows * chunks > kLineThreads || rows * row > 100 * 1024) rows = 4;
  k_adi_rows<<<dim3((most_rows + rows - 1) / rows, count), (rows * chunks + 31) / 32 * 32, rows * row, s>>>(q, rows);
  OFB_LAUNCH_CHECK("k_adi_rows");
}

// Lets every line solver use the shared memory of its longest line.  The
// attribute belongs to the kernel, not to a plan: set to one launch's size it
// would be another thread's launch that fails.
void adi_attributes() {
  constexpr int kMost = 227 * 1024;  // per block, all of it dynamic in these kernels
  auto attr = [](auto kern) {
    OFB_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  };
  attr(k_adi_scan<true, 4>);
  attr(k_adi_scan<false, 4>);
  attr(k_adi_scan<true, 16>);
  attr(k_adi_scan<false, 16>);
  attr(k_adi_tile<true>);
  attr(k_adi_tile<false>);
  attr(k_adi_rows);
}

}  // namespace

void launch_adi_sweeps(const AdiPlan* p, int axis, const double* const* in, double* const* out, cudaStream_t s) {
  int together[3], count = 0;
  for(int c = 0; c < 3; ++c) {
    if(!p->ax[c][axis].active) continue;
    if(p->ax[c][axis].chunked) together[count++] = c;
    else launch_adi_sweep(p, c, axis, in[c], out[c], s);
  }
  if(count > 0) launch_chunked(p, together, count, axis, in, out, s);
}

void launch_adi_sweep(const AdiPlan* p, int comp, int axis, const double* in, double* out,
                      cudaStream_t s) {
  const AdiAxis& A = p->ax[comp][axis];
  if(!A.active) return;
  if(A.chunked) {
    const double* ins[3] = {in, in, in};
    double* outs[3] = {out, out, out};
    launch_chunked(p, &comp, 1, axis, ins, outs, s);
    return;
  }
  SweepArgs a;
  a.L = make_lay(p->g, kFaceX + comp);
  a.axis = axis;
  a.n = A.n;
  a.begin = A.begin;
  a.dup_index = A.dup_index;
  a.periodic = A.periodic ? 1 : 0;
  a.copy_duplicate = A.copy_duplicate ? 1 : 0;
  a.lower = A.lower;
  a.rhs_first = A.rhs_first;
  a.rhs_last = A.rhs_last;
  a.uc_over_gamma = A.uc_over_gamma;
  a.inv_den = A.inv_den;
  a.cu = p->coef + A.off;
  a.ip = p->coef + A.off + A.n;
  a.z = p->coef + A.off + 2 * A.n;
  const int a1 = axis == 0 ? 1 : 0;
  const int a2 = axis == 2 ? 1 : 2;
  ProfScope ps(kKAdi, s);
  if(A.partition) {
    ScanArgs sa;
    sa.K = A.seg;
    const int KP = A.seg * 32;
    const double* base = p->coef + A.poff;
    sa.ip = base;
    sa.fB = base + KP;
    sa.cu = base + 2 * KP;
    sa.gD = base + 3 * KP;
    sa.z = base + 4 * KP;
    sa.mf = base + 5 * KP;
    sa.mb = base + 5 * KP + 5 * 32;
    // 16 lines per block; 4 when that leaves fewer than two blocks per SM
    // (few long lines, e.g. a 2D sweep)
    const long long nl = static_cast<long long>(a.L.n(a1)) * a.L.n(a2);
    if((nl + 15) / 16 >= 2LL * 148)
      launch_scan<16>(a, sa, axis, a1, a2, in, out, s);
    else
      launch_scan<4>(a, sa, axis, a1, a2, in, out, s);
    OFB_LAUNCH_CHECK("k_adi_scan");
    return;
  }
  // lines per warp so that one tile fits kAdiTileBytes (32 when n <= 255)
  int lines = 32;
  while(lines > 1 && static_cast<size_t>(lines) * (a.n + 1) * sizeof(double) > kAdiTileBytes) lines /= 2;
  const size_t smem = static_cast<size_t>(lines) * (a.n + 1) * sizeof(double);
  if(axis == 0) {
    const long long nl = static_cast<long long>(a.L.n(a1)) * a.L.n(a2);
    dim3 grid(static_cast<unsigned>((nl + lines - 1) / lines), 1, 1);
    k_adi_tile<true><<<grid, 32, smem, s>>>(a, in, out, lines);
  } else {
    dim3 grid((a.L.n(a1) + lines - 1) / lines, a.L.n(a2), 1);
    k_adi_tile<false><<<grid, 32, smem, s>>>(a, in, out, lines);
  }
  OFB_LAUNCH_CHECK("k_adi_tile");
}

}  // namespace ofb
