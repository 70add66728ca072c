// Host side of the orientation/shape-averaged observables: orientation
// distribution coefficients, shape distribution nodes, and the get_table
// pipeline (T-matrices -> orientation average -> S -> Q / Z -> shape average).
//
// Reference (CosTuuM): CTMModule.cpp:146-478 (get_table), TaskManager.hpp:
// 445-1346 (the per-grain task graph), OrientationDistribution.hpp:220-243,
// MishchenkoOrientationDistribution.hpp:107-118,
// DavisGreensteinOrientationDistribution.hpp:81-102,
// ShapeDistribution.hpp:95-106, DraineHensleyShapeDistribution.hpp.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "tmx_ctx.h"

// ------------------------------------------------------ quadrature tools --

// Gauss-Legendre rule on [a, b] (get_gauss_legendre_points_and_weights_ab,
// SpecialFunctions.hpp:737-751)
static void gl_ab(int order, double a, double b, double *x, double *w) {
  tmx_host_gauss_legendre(order, x, w);
  const double wfac = 0.5 * (b - a);
  const double xterm = 0.5 * (a + b);
  for (int i = 0; i < order; ++i) {
    x[i] = wfac * x[i] + xterm;
    w[i] *= wfac;
  }
}

// Adaptive Gauss-Legendre quadrature that raises the order by one until
// either the absolute or the relative change is below its target
// (gauss_legendre_quadrature, SpecialFunctions.hpp:771-810).
template <typename F>
static double gl_quadrature(F f, double lower, double upper, int start,
                            int maximum, double abs_tol, double rel_tol) {
  int order = start;
  double old_q = 0.;
  double absd = abs_tol + 1.;
  double reld = rel_tol + 1.;
  std::vector<double> x(maximum > 0 ? maximum : 1), w(x.size());
  while (order < maximum && absd > abs_tol && reld > rel_tol) {
    gl_ab(order, lower, upper, x.data(), w.data());
    double q = 0.;
    for (int i = 0; i < order; ++i) {
      q += w[i] * f(x[i]);
    }
    absd = fabs(q - old_q);
    reld = absd / fabs(q + old_q);
    old_q = q;
    ++order;
  }
  return old_q;
}

// Legendre P_n(cos beta) = d^n_00(beta) by the m = 0 recurrence of
// SpecialFunctions::wigner_dn_0m (SpecialFunctions.hpp:302-371)
static double wigner_d00(double cosx, int order) {
  if (order == 0) {
    return 1.;
  }
  double d1 = 1., d2 = cosx, last = cosx;
  for (int n = 0; n < order; ++n) {
    const double np1 = n + 1.;
    const double np2 = n + 2.;
    const double np12p1 = 2. * np1 + 1.;
    const double dnp1 = (np12p1 * cosx * d2 - np1 * d1) / np2;
    last = d2;
    d1 = d2;
    d2 = dnp1;
  }
  return last;
}

// ------------------------------------------------------- distributions ---

extern "C" int tmx_orientation_coefficients(int kind, double param, int order,
                                            double (*fn)(double, void *),
                                            void *arg, double *out) {
  if (order < 0 || !out || kind < 0 || kind > 3 || (kind == 3 && !fn)) {
    return TMX_ERR_INVALID;
  }
  for (int i = 0; i <= order; ++i) {
    out[i] = 0.;
  }
  if (kind == 1) {
    // Mishchenko: p(beta) = 1/2 + 5/4 p2 (3 cos^2 - 1), p2 = 3/2 <cos^2> - 1/2
    out[0] = 1.;
    if (order >= 2) {
      out[2] = 1.5 * param - 0.5;
    }
    return TMX_OK;
  }
  if (kind == 2) {
    // Davis-Greenstein perfect alignment
    if (param < 1.) {
      double nominator = 1., denominator = 2.;
      out[0] = 1.;
      for (int i = 1; 2 * i < order + 1; ++i) {
        const int sign = (i % 2 == 0) ? 1 : -1;
        out[2 * i] = sign * nominator / denominator;
        nominator *= 2. * i + 1.;
        denominator *= 2. * (i + 1.);
      }
    } else {
      for (int i = 0; i <= order; ++i) {
        out[i] = 1.;
      }
    }
    return TMX_OK;
  }
  // numerical: random (p = 1/2; tolerances 1e-10 / 1e-5) or custom
  // (Python function; tolerances 1e-4 / 1e-4, PyOrientationDistribution.hpp)
  auto p = [&](double beta) { return kind == 0 ? 0.5 : fn(beta, arg); };
  const double at = (kind == 0) ? 1.e-10 : 1.e-4;
  const double rt = (kind == 0) ? 1.e-5 : 1.e-4;
  const double norm = gl_quadrature(
      [&](double beta) { return sin(beta) * p(beta); }, 0., M_PI, 100, 1000,
      at, rt);
  const double nf = 1. / norm;
  out[0] = 1.;
  auto coefficient = [&](int i) {
    return gl_quadrature(
        [&](double beta) {
          const double cb = cos(beta);
          const double sb = sin(beta);
          const double pb = nf * p(beta);
          return sb * pb * wigner_d00(cb, i);
        },
        0., M_PI, 2 * (i + 1), 100 * (i + 1), at, rt);
  };
  // the coefficients are independent quadratures (their cost grows with
  // the order): random orientation spreads them over host threads,
  // interleaved; a custom p(beta) calls into Python and stays on this thread
  if (kind == 0 && order >= 32) {
    const int nt = std::max(
        1, std::min<int>((int)std::thread::hardware_concurrency(), 32));
    std::vector<std::thread> pool;
    int started = 0;
    try {
      for (int t = 0; t < nt; ++t) {
        pool.emplace_back([&, t]() {
          for (int i = 1 + t; i <= order; i += nt) {
            out[i] = coefficient(i);
          }
        });
        ++started;
      }
    } catch (const std::system_error &) {
      // fewer threads than asked for: the residues of the missing ones below
    }
    for (std::thread &th : pool) {
      th.join();
    }
    for (int t = started; t < nt; ++t) {
      for (int i = 1 + t; i <= order; i += nt) {
        out[i] = coefficient(i);
      }
    }
    return TMX_OK;
  }
  for (int i = 1; i <= order; ++i) {
    out[i] = coefficient(i);
  }
  return TMX_OK;
}

namespace {

// DraineHensleyShapeDistribution helpers (DraineHensleyShapeDistribution.hpp)
double dh_shape_factor(double d) {
  if (d < 1.) {
    const double e2 = 1. - d * d;
    const double e = sqrt(e2);
    return (1. - e2) * (0.5 * log((1. + e) / (1. - e)) / e - 1.) / e2;
  } else if (d > 1.) {
    const double e2 = 1. - 1. / (d * d);
    const double e = sqrt(e2);
    return (1. - sqrt(1. - e2) * asin(e) / e) / e2;
  }
  return 1. / 3.;
}

double dh_jacobian(double d) {
  if (d < 1.) {
    const double e2 = 1. - d * d;
    if (e2 < 1.e-5) {
      return 4. / 15. + 2. * e2 / 21. + 3. * e2 * e2 / 70.;
    }
    const double e = sqrt(e2);
    return 0.5 * sqrt(1. - e2) * ((3. - e2) * log((1. + e) / (1. - e)) - 6. * e) /
           (e2 * e2 * e);
  } else if (d > 1.) {
    const double e2 = 1. - 1. / (d * d);
    if (e2 < 1.e-5) {
      return 4. / 15. - 2. * e2 / 21. - 11. * e2 * e2 / 210.;
    }
    const double e = sqrt(e2);
    return (1. - e2) * ((3. - 2. * e2) * asin(e) - 3. * e * sqrt(1. - e2)) /
           (e2 * e2 * e);
  }
  return 4. / 15.;
}

double dh_cde2(double L) {
  const double Lm1 = L - 1.;
  return 12. * L * Lm1 * Lm1;
}

double dh_eval(double d) { return dh_cde2(dh_shape_factor(d)) * dh_jacobian(d); }

} // namespace

// kind 0: the default ShapeDistribution (exp(-(d-1)^2 / (2 x 0.027777778))
// on [0.5, 1.5]); kind 1: Draine & Hensley (2017) CDE2 with a probability
// cutoff (param1) or a prolate/oblate fraction (param2 > 0)
extern "C" int tmx_shape_distribution(int kind, int npoints, double param1,
                                      double param2, double *shapes,
                                      double *weights, double *limits) {
  if (npoints < 1 || !shapes || !weights || kind < 0 || kind > 1) {
    return TMX_ERR_INVALID;
  }
  double dmin = 0.5, dmax = 1.5;
  auto pdf = [&](double d) -> double {
    if (kind == 0) {
      if (d >= 0.5 && d <= 1.5) {
        const double x = d - 1.;
        return exp(-0.5 * x * x / 0.027777778);
      }
      return 0.;
    }
    return (d >= dmin && d <= dmax) ? dh_eval(d) : 0.;
  };
  if (kind == 1) {
    const double cutoff = param1, fraction = param2;
    if (fraction > 0.) {
      auto integ = [&](double a, double b) {
        return gl_quadrature([&](double d) { return dh_eval(d); }, a, b, 10,
                             1000, 1.e-10, 1.e-10);
      };
      const double prolate_fraction = integ(0., 1.);
      const double prolate_target = fraction * prolate_fraction;
      double lower = 0., upper = 1., half = 0.5;
      double integral = integ(half, 1.);
      int guard = 0;
      while (fabs(integral - prolate_target) >
                 0.005 * fabs(integral + prolate_target) &&
             ++guard < 200) {
        if (integral > prolate_target) {
          lower = half;
        } else {
          upper = half;
        }
        half = 0.5 * (lower + upper);
        integral = integ(half, 1.);
      }
      dmin = half;
      const double oblate_target = fraction * (1. - prolate_fraction);
      lower = 1.;
      upper = 2.;
      integral = integ(1., upper);
      guard = 0;
      while (integral < oblate_target && ++guard < 60) {
        upper *= 2.;
        integral = integ(1., upper);
      }
      half = 0.5 * (lower + upper);
      integral = integ(1., half);
      guard = 0;
      while (fabs(integral - oblate_target) > 1.e-5 * fabs(integral + oblate_target) &&
             ++guard < 200) {
        if (integral > oblate_target) {
          upper = half;
        } else {
          lower = half;
        }
        half = 0.5 * (lower + upper);
        integral = integ(1., half);
      }
      dmax = half;
    } else {
      dmin = 1.;
      dmax = 1.;
      double valmin = pdf(dmin) - cutoff;
      int guard = 0;
      while (valmin > 0. && ++guard < 200) {
        dmin *= 0.5;
        valmin = pdf(dmin) - cutoff;
      }
      double ub = 1.;
      guard = 0;
      while (fabs(dmin - ub) > 0.005 * fabs(dmin + ub) && ++guard < 200) {
        const double mid = 0.5 * (dmin + ub);
        const double v = pdf(mid) - cutoff;
        if (v < 0.) {
          dmin = mid;
        } else {
          ub = mid;
        }
      }
      double valmax = pdf(dmax) - cutoff;
      guard = 0;
      while (valmax > 0. && ++guard < 1000) {
        dmax += 1.;
        valmax = pdf(dmax) - cutoff;
      }
      double lb = 1.;
      guard = 0;
      while (fabs(dmax - lb) > 0.005 * fabs(dmax + lb) && ++guard < 200) {
        const double mid = 0.5 * (lb + dmax);
        const double v = pdf(mid) - cutoff;
        if (v > 0.) {
          lb = mid;
        } else {
          dmax = mid;
        }
      }
    }
  }
  if (limits) {
    limits[0] = dmin;
    limits[1] = dmax;
  }
  // ShapeDistribution::evaluate: GL nodes on [dmin, dmax], weight x p(d)
  gl_ab(npoints, dmin, dmax, shapes, weights);
  for (int i = 0; i < npoints; ++i) {
    weights[i] *= pdf(shapes[i]);
  }
  return TMX_OK;
}

// R_V / R_S of a spheroid (get_equal_volume_to_equal_surface_area_sphere_
// ratio, SpecialFunctions.hpp:557-583)
extern "C" double tmx_rv_over_rs(double d) {
  if (d > 1.) {
    const double d2 = d * d;
    const double e = sqrt(1. - 1. / d2);
    const double cbrtd2 = cbrt(d2);
    return 1. / sqrt(0.25 * (2. * cbrtd2 +
                             log((1. + e) / (1. - e)) / (e * cbrtd2 * cbrtd2)));
  } else if (d < 1.) {
    const double cbrtd = cbrt(d);
    const double e = sqrt(1. - d * d);
    return 1. / sqrt(0.5 * (cbrtd * cbrtd + asin(e) / (e * cbrtd)));
  }
  return 1.;
}

// -------------------------------------------------------------- get_table --

namespace {

// zenith angle as the reference's grids compute it
TmxAngle make_angle(double cost) {
  TmxAngle a;
  a.c = cost;
  a.s = sqrt((1. - cost) * (1. + cost));
  a.si = (a.s != 0.) ? 1. / a.s : 9000.;
  return a;
}

int64_t est_nmax(double x, int min_order, int max_order) {
  double e = x + 4.05 * cbrt(x) + 8.;
  e = std::max<double>(e, min_order);
  return std::min<int64_t>((int64_t)e, max_order - 1);
}

// one amplitude job: an incoming and an outgoing angle, nphi azimuths from
// phi0 on, the first S at out
struct AmpJob {
  int32_t ain, aout, nphi;
  int64_t phi0, out;
};

// groups of a set of jobs (TmxAmpGroup without a grain): by distinct incoming
// angle in order of first use, at most TMX_AMP_NIN of them and about
// kGroupPairs pairs per group. The pi and tau columns of the plan's angles (16
// bytes per order and block m of each) are in memory kColumnBytes at a time:
// where the angles need more, the groups go in passes, each with the angles it
// uses renumbered, and an angle that several passes use has its columns made in
// each of them (a column costs as much as one product with one).
struct AmpPlan {
  static constexpr int kGroupPairs = 512;
  static constexpr int64_t kColumnBytes = (int64_t)512 << 20;
  struct Pass {
    int g0, g1;     // groups
    int64_t a0, na; // angles
  };
  std::vector<int32_t> ins;
  std::vector<TmxAmpPair> pairs;
  std::vector<TmxAmpGroup> groups;
  std::vector<Pass> passes;
  std::vector<int32_t> angles; // angle of each number of each pass, if split
  bool split;

  // nang angles in all, orders of at most nmax
  AmpPlan(int64_t nang, int nmax)
      : split(nang > pass_angles(nmax)), nang_(nang), cap_(pass_angles(nmax)) {
    if (split) {
      number_.resize(nang);
      number_pass_.assign(nang, -1);
    }
    slot_.assign(nang, -1);
    passes.push_back({0, 0, 0, split ? 0 : nang});
  }

  // (a group's angles always fit a pass)
  static int64_t pass_angles(int nmax) {
    return std::max<int64_t>(kGroupPairs + TMX_AMP_NIN + 1,
                             kColumnBytes / (16 * (int64_t)(nmax + 1) * nmax));
  }

  // returns the new groups [first, second) of n jobs, the j-th being job(j)
  template <class Job> std::pair<int, int> add(int32_t n, Job job) {
    const int g0 = (int)groups.size();
    // jobs by incoming angle: a stable counting sort, left out where they come
    // in that order
    start_.assign(1, 0);
    start_.reserve((size_t)n + 1);
    first_.clear();
    first_.reserve(n);
    bool in_order = true;
    for (int32_t j = 0; j < n; ++j) {
      const int32_t a = job(j).ain;
      int32_t &s = slot_[a];
      if (s < 0) {
        s = (int32_t)first_.size();
        first_.push_back(a);
        start_.push_back(0);
      }
      in_order = in_order && s + 1 == (int32_t)first_.size();
      ++start_[s + 1];
    }
    for (size_t a = 1; a < start_.size(); ++a) {
      start_[a] += start_[a - 1];
    }
    if (!in_order) {
      sorted_.resize(n);
      pos_.assign(start_.begin(), start_.end() - 1);
      for (int32_t j = 0; j < n; ++j) {
        sorted_[pos_[slot_[job(j).ain]]++] = j;
      }
    }
    if (pairs.empty()) {
      pairs.reserve(n);
      ins.reserve(first_.size());
    }
    TmxAmpGroup g = {};
    const auto close_group = [&]() {
      if (g.npair > 0) {
        number(g);
        groups.push_back(g);
        passes.back().g1 = (int)groups.size();
      }
      g = TmxAmpGroup{};
    };
    for (size_t a = 0; a < first_.size(); ++a) {
      for (int32_t q = start_[a]; q < start_[a + 1]; ++q) {
        const AmpJob J = job(in_order ? q : sorted_[q]);
        const bool fresh = q == start_[a];
        if (g.npair >= kGroupPairs || (fresh && g.nin == TMX_AMP_NIN)) {
          close_group();
        }
        if (g.npair == 0) {
          g.in0 = (int32_t)ins.size();
          g.pair0 = (int32_t)pairs.size();
        }
        if (fresh || g.nin == 0) {
          ins.push_back(J.ain);
          ++g.nin;
        }
        TmxAmpPair p;
        p.in = g.nin - 1;
        p.angle_out = J.aout;
        p.nphi = J.nphi;
        p.pref = g.nitem;
        p.phi0 = J.phi0;
        p.out = J.out;
        pairs.push_back(p);
        ++g.npair;
        g.nitem += p.nphi;
      }
    }
    close_group();
    for (int32_t a : first_) {
      slot_[a] = -1;
    }
    return {g0, (int)groups.size()};
  }
  std::pair<int, int> add(const std::vector<AmpJob> &jobs) {
    return add((int32_t)jobs.size(), [&](int32_t j) { return jobs[j]; });
  }

private:
  // the group's angles by their numbers in its pass, a new one if they do not
  // fit the present one
  void number(const TmxAmpGroup &g) {
    if (!split) {
      return;
    }
    const int64_t before = (int64_t)angles.size();
    const auto see = [&](int32_t a) {
      if (number_pass_[a] != (int32_t)passes.size()) {
        number_pass_[a] = (int32_t)passes.size();
        number_[a] = (int32_t)((int64_t)angles.size() - passes.back().a0);
        angles.push_back(a);
      }
    };
    const auto see_all = [&]() {
      for (int32_t k = 0; k < g.nin; ++k) {
        see(ins[g.in0 + k]);
      }
      for (int32_t k = 0; k < g.npair; ++k) {
        see(pairs[g.pair0 + k].angle_out);
      }
    };
    see_all();
    if ((int64_t)angles.size() - passes.back().a0 > cap_) {
      angles.resize(before);
      const int n = (int)groups.size();
      passes.push_back({n, n, before, 0});
      see_all();
    }
    passes.back().na = (int64_t)angles.size() - passes.back().a0;
    for (int32_t k = 0; k < g.nin; ++k) {
      ins[g.in0 + k] = number_[ins[g.in0 + k]];
    }
    for (int32_t k = 0; k < g.npair; ++k) {
      int32_t &a = pairs[g.pair0 + k].angle_out;
      a = number_[a];
    }
  }

  int64_t nang_, cap_;
  std::vector<int32_t> slot_, first_, number_, number_pass_, start_, pos_, sorted_;
};

// groups [g0, g1) of a plan for one grain, their S from out0 on
struct AmpUse {
  int32_t grain;
  int g0, g1;
  int64_t out0;
};

// Work plan of the observable kernels for the grains `og` (already on the
// device in ctx->o_og): the orientation kernel's pair-major order and the
// amplitude kernel's groups of every grain (`uses`, by descending order) in
// launches of blocks of similar size. ang: the angles the plan's jobs name.
int upload_obs_plan(tmx_ctx *ctx, const std::vector<TmxObsGrain> &og,
                    const std::vector<TmxAngle> &ang, const AmpPlan &plan,
                    std::vector<AmpUse> uses) {
  int rc0;
  ++ctx->plan_seq;
  cudaStream_t st = ctx->stream;
  const int64_t n = (int64_t)og.size();
  // orientation-average work items (tmx_launch_orient): grains by descending
  // order, so that those of order >= n are the first at_least[n]
  int nbmax = 1;
  for (int64_t g = 0; g < n; ++g) {
    nbmax = std::max(nbmax, og[g].nmax);
  }
  std::vector<int32_t> order;
  for (int64_t g = 0; g < n; ++g) {
    if (og[g].nmax > 0) {
      order.push_back((int32_t)g);
    }
  }
  std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
    return og[a].nmax > og[b].nmax;
  });
  std::vector<int64_t> at_least(nbmax + 2, 0); // grains of order >= k
  for (int32_t g : order) {
    at_least[og[g].nmax] += 1;
  }
  for (int k = nbmax; k >= 1; --k) {
    at_least[k] += at_least[k + 1];
  }
  // one launch per range of n = max(n1, n2), largest first: shared memory is
  // sized by the range, and so is the chunk of grains per warp -- eight where
  // their rows leave room for a dozen warps per SM (n < 32), four above, and
  // no more than there are grains (idle columns cost as much as used ones)
  std::vector<TmxOrientRange> orng;
  ctx->o_orient.clear();
  const int oedge[] = {TMX_MAX_NB, 63, 31, 15, 0}; // M + 1 rows in tiles of 8
  for (int b = 0; b < 4; ++b) {
    tmx_ctx::OrientLaunch la;
    la.rng0 = (int)orng.size();
    const int top = std::min(oedge[b], nbmax);
    const int64_t most = (top > oedge[b + 1]) ? at_least[oedge[b + 1] + 1] : 0;
    la.chunk = most <= 2 ? 2 : (most <= 4 || oedge[b] > 31) ? 4 : 8;
    la.ncap = top;
    for (int nn = top; nn > oedge[b + 1]; --nn) {
      if (at_least[nn] > 0) {
        orng.push_back({la.nitems, nn, (int32_t)at_least[nn]});
        la.nitems += (2 * nn - 1) * ((at_least[nn] + la.chunk - 1) / la.chunk);
      }
    }
    la.nrng = (int)orng.size() - la.rng0;
    if (la.nitems > 0) {
      ctx->o_orient.push_back(la);
    }
  }
  if ((rc0 = ensure(ctx, ctx->o_ord, std::max<size_t>(1, order.size()) * sizeof(int32_t)))) {
    return rc0;
  }
  if (!order.empty()) {
    CK(cudaMemcpyAsync(ctx->o_ord.p, order.data(), order.size() * sizeof(int32_t),
                       cudaMemcpyHostToDevice, st));
  }
  uses.erase(std::remove_if(uses.begin(), uses.end(),
                            [&](const AmpUse &u) { return og[u.grain].nmax <= 0; }),
             uses.end());
  std::stable_sort(uses.begin(), uses.end(), [&](const AmpUse &a, const AmpUse &b) {
    return og[a.grain].nmax > og[b.grain].nmax;
  });
  std::vector<TmxAmpGroup> grp;
  std::vector<size_t> pass_end; // groups of the passes, one after the other
  for (const AmpPlan::Pass &p : plan.passes) {
    for (const AmpUse &u : uses) {
      for (int k = std::max(u.g0, p.g0); k < std::min(u.g1, p.g1); ++k) {
        TmxAmpGroup g = plan.groups[k];
        g.grain = u.grain;
        g.out0 = u.out0;
        grp.push_back(g);
      }
    }
    pass_end.push_back(grp.size());
  }
  // chunks of groups whose m sums fit the X buffer, and per chunk one launch
  // per block size: ranges of groups whose block m has lo < L <= hi orders
  ctx->o_chunks.clear();
  std::vector<TmxAmpRange> rng;
  const int64_t x_cap = (int64_t)1 << 24; // complex elements per matrix
  int64_t x_max = 1;
  int pass = 0;
  for (size_t g0 = 0; g0 < grp.size();) {
    while (g0 >= pass_end[pass]) {
      ++pass;
    }
    tmx_ctx::AmpChunk ch;
    ch.g0 = (int)g0;
    ch.pass = pass;
    int64_t x = 0;
    size_t g1 = g0;
    for (; g1 < pass_end[pass]; ++g1) {
      const int64_t need = (int64_t)grp[g1].npair * (og[grp[g1].grain].nmax + 1) * 4;
      if (g1 > g0 && x + need > x_cap) {
        break;
      }
      grp[g1].x0 = x;
      x += need;
      ch.nitem_max = std::max(ch.nitem_max, grp[g1].nitem);
      ch.nin = std::max(ch.nin, grp[g1].nin);
    }
    ch.g1 = (int)g1;
    x_max = std::max(x_max, x);
    const int top = og[grp[g0].grain].nmax;
    // groups of the chunk of order >= k are its first at(k)
    std::vector<int> at(top + 2, 0);
    for (size_t g = g0; g < g1; ++g) {
      at[og[grp[g].grain].nmax] += 1;
    }
    for (int k = top - 1; k >= 0; --k) {
      at[k] += at[k + 1];
    }
    const int edges[] = {TMX_MAX_NB, 64, 32, 16, 0};
    for (int b = 0; b < 4; ++b) {
      const int hi = edges[b], lo = edges[b + 1];
      tmx_ctx::AmpLaunch la;
      la.rng0 = (int)rng.size();
      for (int m = 0; m <= top; ++m) {
        // L = N + 1 - max(m, 1): orders nlo .. nhi
        const int nlo = std::max(m, 1) + lo, nhi = std::max(m, 1) - 1 + hi;
        const int first = nhi + 1 <= top ? at[nhi + 1] : 0;
        const int last = nlo <= top ? at[nlo] : 0;
        if (last > first) {
          rng.push_back({la.nitems, m, ch.g0 + first});
          la.nitems += last - first;
          la.lcap = std::max(la.lcap, std::min(hi, top + 1 - std::max(m, 1)));
        }
      }
      la.nrng = (int)rng.size() - la.rng0;
      if (la.nitems > 0) {
        ch.launches.push_back(la);
      }
    }
    ctx->o_chunks.push_back(ch);
    g0 = g1;
  }
  int rc;
  const auto put = [&](DevBuf &buf, const void *src, size_t bytes) -> int {
    const int r = ensure(ctx, buf, std::max<size_t>(16, bytes));
    if (r || bytes == 0) {
      return r;
    }
    CK(cudaMemcpyAsync(buf.p, src, bytes, cudaMemcpyHostToDevice, st));
    return TMX_OK;
  };
  // angles of the passes, one after the other
  std::vector<TmxAngle> by_pass;
  for (int32_t a : plan.angles) {
    by_pass.push_back(ang[a]);
  }
  const std::vector<TmxAngle> &table = plan.split ? by_pass : ang;
  ctx->o_passes.clear();
  for (const AmpPlan::Pass &p : plan.passes) {
    ctx->o_passes.push_back({p.a0, p.na});
  }
  if ((rc = put(ctx->o_angles, table.data(), table.size() * sizeof(TmxAngle))) ||
      (rc = put(ctx->o_orng, orng.data(), orng.size() * sizeof(TmxOrientRange))) ||
      (rc = put(ctx->o_grp, grp.data(), grp.size() * sizeof(TmxAmpGroup))) ||
      (rc = put(ctx->o_ins, plan.ins.data(), plan.ins.size() * sizeof(int32_t))) ||
      (rc = put(ctx->o_prs, plan.pairs.data(), plan.pairs.size() * sizeof(TmxAmpPair))) ||
      (rc = put(ctx->o_rng, rng.data(), rng.size() * sizeof(TmxAmpRange)))) {
    return rc;
  }
  CK(cudaStreamSynchronize(st));
  ctx->o_nbmax = nbmax;
  ctx->o_xcap = x_max;
  if (ctx->profiling) {
    // flops of one matrix set over the kernels' index spaces: the
    // orientation average 16 (M + 1)^2 per (n1, n2), M = min(n1, n2),
    // of every averaged grain; the amplitudes 16 L^2 per m block (L orders)
    // and incoming angle and 32 L per pair
    double fo = 0., fa = 0.;
    for (int64_t g = 0; g < n; ++g) {
      const int N = og[g].nmax;
      if (N > 0 && og[g].coef_set >= 0) {
        for (int a = 1; a <= N; ++a) {
          for (int b = 1; b <= N; ++b) {
            const double M = std::min(a, b);
            fo += 16. * (M + 1.) * (M + 1.);
          }
        }
      }
    }
    for (const TmxAmpGroup &g : grp) {
      const int N = og[g.grain].nmax;
      for (int m = 0; m <= N; ++m) {
        const double L = N + 1 - std::max(m, 1);
        fa += 16. * L * L * g.nin + 32. * L * g.npair;
      }
    }
    ctx->o_fl_orient = fo;
    ctx->o_fl_amp = fa;
  }
  return TMX_OK;
}

// the plan's orientation launches on ctx->stream
int launch_orient(tmx_ctx *ctx, const TmxMatSet &mats, int nmat, int ncoef, int fold) {
  for (const tmx_ctx::OrientLaunch &la : ctx->o_orient) {
    tmx_launch_orient((const TmxObsGrain *)ctx->o_og.p, (const int32_t *)ctx->o_ord.p,
                      (const TmxOrientRange *)ctx->o_orng.p + la.rng0, la.nrng, la.nitems,
                      la.ncap, la.chunk, mats, nmat, (const double *)ctx->o_coef.p, ncoef,
                      (const int64_t *)ctx->cg_off.p, (const double *)ctx->cg.p,
                      ctx->cg_nmax, fold, ctx->stream);
    LAUNCHED();
  }
  return TMX_OK;
}

// Ta = orientation average (or copy) of Tsrc with the amplitude factors
// folded in (compact class layout), then the amplitudes S of every job (zeroed first: grains with
// nmax 0 have no jobs)
int run_amplitudes(tmx_ctx *ctx, const cplx *const *Tsrc, int nmat,
                   int64_t t_total, int ncoef, cplx *const *S_out,
                   int64_t s_total) {
  cudaStream_t st = ctx->stream;
  int rc;
  // (t_total is even: every T-matrix has a multiple of four elements)
  const int64_t ta_total = (t_total + 1) / 2;
  if ((rc = ensure(ctx, ctx->Ta,
                   std::max<int64_t>(1, nmat * ta_total) * sizeof(cplx)))) {
    return rc;
  }
  for (int k = 0; k < nmat; ++k) {
    CK(cudaMemsetAsync(S_out[k], 0, std::max<int64_t>(0, s_total) * 4 * sizeof(cplx),
                       st));
  }
  if (t_total <= 0 || ctx->o_orient.empty()) {
    return TMX_OK;
  }
  TmxMatSet avg = {}, amp = {};
  for (int k = 0; k < nmat; ++k) {
    avg.src[k] = Tsrc[k];
    avg.dst[k] = (cplx *)ctx->Ta.p + k * ta_total;
    amp.src[k] = avg.dst[k];
    amp.dst[k] = S_out[k];
  }
  if ((rc = ensure(ctx, ctx->o_x, (size_t)nmat * ctx->o_xcap * sizeof(cplx)))) {
    return rc;
  }
  cudaEvent_t pe = nullptr;
  if ((rc = prof_begin(ctx, TMX_PROF_ORIENT, &pe))) {
    return rc;
  }
  if ((rc = launch_orient(ctx, avg, nmat, ncoef, 1))) {
    return rc;
  }
  // T-matrices in and averaged T-matrices (compact, half the size) out
  if ((rc = prof_end(ctx, TMX_PROF_ORIENT, pe, nmat * ctx->o_fl_orient, st,
                     1.5 * nmat * t_total * sizeof(cplx)))) {
    return rc;
  }
  if ((rc = prof_begin(ctx, TMX_PROF_AMP, &pe))) {
    return rc;
  }
  // the pi / tau columns of the angles of a pass, once for all grains
  const int wn = ctx->o_nbmax;
  int64_t na = 0;
  for (const auto &p : ctx->o_passes) {
    na = std::max(na, p[1]);
  }
  const size_t wcol = (size_t)na * (wn + 1) * wn;
  if ((rc = ensure(ctx, ctx->o_wcol, std::max<size_t>(1, 2 * wcol) * sizeof(double)))) {
    return rc;
  }
  double *wpi = (double *)ctx->o_wcol.p, *wtau = wpi + wcol;
  const TmxAmpGroup *grp = (const TmxAmpGroup *)ctx->o_grp.p;
  const TmxAmpPair *prs = (const TmxAmpPair *)ctx->o_prs.p;
  const TmxObsGrain *og = (const TmxObsGrain *)ctx->o_og.p;
  int pass = -1;
  for (const tmx_ctx::AmpChunk &ch : ctx->o_chunks) {
    if (ch.pass != pass) {
      pass = ch.pass;
      tmx_launch_wigner_cols((const TmxAngle *)ctx->o_angles.p + ctx->o_passes[pass][0],
                             (int)ctx->o_passes[pass][1], wn, wpi, wtau, st);
      LAUNCHED();
    }
    for (const tmx_ctx::AmpLaunch &la : ch.launches) {
      tmx_launch_amp(grp, (const int32_t *)ctx->o_ins.p, prs,
                     (const TmxAmpRange *)ctx->o_rng.p + la.rng0, la.nrng, la.nitems,
                     og, amp, nmat, wpi, wtau, wn, (cplx *)ctx->o_x.p, ctx->o_xcap,
                     la.lcap, ch.nin, st);
      LAUNCHED();
    }
    tmx_launch_azimuth(grp + ch.g0, ch.g1 - ch.g0, prs, og, amp, nmat,
                       (const cplx *)ctx->o_phis.p, (const cplx *)ctx->o_x.p,
                       ctx->o_xcap, ch.nitem_max, st);
    LAUNCHED();
  }
  // averaged T-matrices in, four complex amplitudes per pair and azimuth out
  if ((rc = prof_end(ctx, TMX_PROF_AMP, pe, nmat * ctx->o_fl_amp, st,
                     nmat * (t_total / 2. + 4. * s_total) * sizeof(cplx)))) {
    return rc;
  }
  return TMX_OK;
}

int run_amplitudes(tmx_ctx *ctx, const cplx *Tsrc, int64_t t_total, int ncoef,
                   cplx *S_out, int64_t s_total) {
  return run_amplitudes(ctx, &Tsrc, 1, t_total, ncoef, &S_out, s_total);
}

} // namespace

extern "C" int tmx_get_table(
    tmx_ctx *ctx, int32_t ntypes, int32_t nsizes, const double *sizes,
    int32_t nlambda, const double *lambdas, int32_t ntheta,
    const double *thetas, int32_t nshape, const double *shapes,
    const double *shape_weights, const double *mr, const double *mi,
    const int32_t *orient_set, int32_t nsets, const double *coeffs,
    int32_t ncoef, int32_t flags, int32_t ngauss, const tmx_schedule *sched,
    double *out_q, double *out_z, int32_t *grain_status) {
  if (!ctx) {
    return TMX_ERR_INVALID;
  }
  const bool do_abs = flags & TMX_TABLE_ABSORPTION;
  const bool do_ext = flags & TMX_TABLE_EXTINCTION;
  const bool do_sca = flags & TMX_TABLE_SCATTERING;
  const bool account = (flags & TMX_TABLE_ACCOUNT_FOR_SCATTERING) && do_abs;
  if (ntypes < 0 || nsizes < 0 || nlambda < 0 || ntheta < 0 || nshape < 1 ||
      !sizes || !lambdas || (ntheta > 0 && !thetas) || !shapes ||
      !shape_weights || !mr || !mi || !orient_set || nsets < 0 ||
      (nsets > 0 && (!coeffs || ncoef < 1)) || (account && ngauss < 1) ||
      ((do_abs || do_ext) && !out_q) || (do_sca && !out_z)) {
    return fail(ctx, TMX_ERR_INVALID, "tmx_get_table: invalid arguments");
  }
  tmx_schedule S = {10, 100, 2, 0, 1.e-4};
  if (sched) {
    S = *sched;
  }
  for (int i = 0; i < nsizes * nshape; ++i) {
    if (orient_set[i] >= nsets) {
      return fail(ctx, TMX_ERR_INVALID, "tmx_get_table: orientation set index");
    }
  }
  const int nq = (do_abs ? 2 : 0) + (do_ext ? 3 : 0);
  const int nphi_sca = 2 * ntheta;
  const int64_t ncells = (int64_t)ntypes * nsizes * nlambda;
  if (ncells == 0 || ntheta == 0 || (!do_abs && !do_ext && !do_sca)) {
    return TMX_OK;
  }
  CK(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  int rc;
  NvtxRange range("tmx_get_table");

  // ---- angle and azimuth tables
  std::vector<TmxAngle> ang;
  for (int i = 0; i < ntheta; ++i) {
    ang.push_back(make_angle(cos(thetas[i])));
  }
  const int acc_a0 = (int)ang.size();
  std::vector<double> acc_w; // [theta weights (ngauss), phi weights (ngauss)]
  std::vector<cplx> phis;
  phis.push_back(mkc(1., 0.)); // azimuth 0 for the theta -> theta amplitude
  int64_t acc_p0 = 0, sca_p0 = 0;
  if (account) {
    std::vector<double> ct(ngauss), wt(ngauss), ph(ngauss), wp(ngauss);
    tmx_host_gauss_legendre(ngauss, ct.data(), wt.data());
    gl_ab(ngauss, 0., 2. * M_PI, ph.data(), wp.data());
    for (int i = 0; i < ngauss; ++i) {
      ang.push_back(make_angle(ct[i]));
    }
    acc_w = wt;
    acc_w.insert(acc_w.end(), wp.begin(), wp.end());
    acc_p0 = (int64_t)phis.size();
    for (int i = 0; i < ngauss; ++i) {
      phis.push_back(mkc(cos(ph[i]), -sin(ph[i])));
    }
  }
  int sca_ain = -1, sca_a0 = -1;
  if (do_sca) {
    sca_ain = (int)ang.size();
    ang.push_back(make_angle(cos(M_PI_2)));
    sca_a0 = (int)ang.size();
    std::vector<double> ct(ntheta), wt(ntheta), ph(nphi_sca), wp(nphi_sca);
    tmx_host_gauss_legendre(ntheta, ct.data(), wt.data());
    for (int i = 0; i < ntheta; ++i) {
      // theta_out = acos(GL node); the grid keeps cos(theta_out) = node
      ang.push_back(make_angle(ct[i]));
    }
    gl_ab(nphi_sca, 0., 2. * M_PI, ph.data(), wp.data());
    sca_p0 = (int64_t)phis.size();
    for (int i = 0; i < nphi_sca; ++i) {
      phis.push_back(mkc(cos(ph[i]), sin(ph[i])));
    }
  }
  if ((rc = ensure(ctx, ctx->o_phis, phis.size() * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->o_wts, std::max<size_t>(1, acc_w.size()) * sizeof(double))) ||
      (rc = ensure(ctx, ctx->o_coef, std::max<int64_t>(1, (int64_t)nsets * ncoef) * sizeof(double))) ||
      (rc = ensure(ctx, ctx->o_shw, nshape * sizeof(double)))) {
    return rc;
  }
  ++ctx->plan_seq; // the observable buffers change below
  CK(cudaMemcpyAsync(ctx->o_phis.p, phis.data(), phis.size() * sizeof(cplx),
                     cudaMemcpyHostToDevice, st));
  if (!acc_w.empty()) {
    CK(cudaMemcpyAsync(ctx->o_wts.p, acc_w.data(), acc_w.size() * sizeof(double),
                       cudaMemcpyHostToDevice, st));
  }
  if (nsets > 0) {
    CK(cudaMemcpyAsync(ctx->o_coef.p, coeffs, (int64_t)nsets * ncoef * sizeof(double),
                       cudaMemcpyHostToDevice, st));
  }
  CK(cudaMemcpyAsync(ctx->o_shw.p, shape_weights, nshape * sizeof(double),
                     cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st)); // host vectors above are about to change

  // ---- chunks of whole cells (all shapes of a cell stay together)
  const int64_t per_grain_s =
      ntheta + (account ? (int64_t)ntheta * ngauss * ngauss : 0) +
      (do_sca ? (int64_t)ntheta * nphi_sca : 0);
  const double budget = 6.e9; // bytes for T, Ta and S of one chunk
  std::vector<double> gr_r, gr_l, gr_mr, gr_mi, gr_d;
  int64_t c0 = 0;
  while (c0 < ncells) {
    // grow the chunk until the estimated memory reaches the budget
    int64_t c1 = c0;
    double bytes = 0.;
    while (c1 < ncells) {
      const int64_t isz = (c1 / nlambda) % nsizes;
      const int64_t il = c1 % nlambda;
      double cell = 0.;
      for (int s = 0; s < nshape; ++s) {
        const double x = 2. * M_PI * sizes[isz] / lambdas[il] * std::max(1., cbrt(shapes[s]));
        const int64_t N = est_nmax(x, S.min_order, S.max_order);
        cell += 2. * tmx_tmatrix_size((int32_t)N) * 16. + per_grain_s * 64.;
      }
      if (c1 > c0 && bytes + cell > budget) {
        break;
      }
      bytes += cell;
      ++c1;
      if ((c1 - c0) * nshape >= 32768) {
        break;
      }
    }
    const int64_t nc = c1 - c0;
    const int64_t ng = nc * nshape;
    gr_r.resize(ng);
    gr_l.resize(ng);
    gr_mr.resize(ng);
    gr_mi.resize(ng);
    gr_d.resize(ng);
    for (int64_t c = 0; c < nc; ++c) {
      const int64_t cell = c0 + c;
      const int64_t isz = (cell / nlambda) % nsizes;
      const int64_t il = cell % nlambda;
      for (int s = 0; s < nshape; ++s) {
        const int64_t g = c * nshape + s;
        gr_r[g] = sizes[isz];
        gr_l[g] = lambdas[il];
        gr_mr[g] = mr[cell];
        gr_mi[g] = mi[cell];
        gr_d[g] = shapes[s];
      }
    }
    if ((rc = tmx_batch_upload(ctx, ng, gr_r.data(), gr_l.data(), gr_mr.data(),
                               gr_mi.data(), gr_d.data(), &S)) ||
        (rc = tmx_batch_compute(ctx))) {
      return rc;
    }
    if (grain_status) {
      for (int64_t g = 0; g < ng; ++g) {
        grain_status[c0 * nshape + g] = ctx->status_h[g];
      }
    }
    // ---- per-grain observable descriptors
    int nmax_chunk = 1;
    std::vector<TmxObsGrain> og(ng);
    int64_t t_total = 0;
    for (int64_t g = 0; g < ng; ++g) {
      const int64_t cell = c0 + g / nshape;
      const int64_t isz = (cell / nlambda) % nsizes;
      const int s = (int)(g % nshape);
      og[g].nmax = ctx->nmax_h[g];
      og[g].coef_set = orient_set[isz * nshape + s];
      og[g].t_off = ctx->t_off_h[g];
      og[g].k = 2. * M_PI / lambdas[cell % nlambda];
      og[g].r_ev = sizes[isz];
      nmax_chunk = std::max(nmax_chunk, og[g].nmax);
      if (og[g].nmax > 0) {
        t_total = std::max<int64_t>(t_total, og[g].t_off + tmx_tmatrix_size(og[g].nmax));
      }
      if (og[g].coef_set >= 0 && 2 * og[g].nmax + 1 > ncoef) {
        return fail(ctx, TMX_ERR_INVALID,
                    "tmx_get_table: orientation coefficients shorter than 2 nmax + 1");
      }
    }
    if ((rc = tmx_ensure_cg(ctx, nmax_chunk))) {
      return rc;
    }
    if ((rc = ensure(ctx, ctx->o_og, ng * sizeof(TmxObsGrain)))) {
      return rc;
    }
    ++ctx->plan_seq; // the observable buffers change below
    CK(cudaMemcpyAsync(ctx->o_og.p, og.data(), ng * sizeof(TmxObsGrain),
                       cudaMemcpyHostToDevice, st));
    // ---- amplitudes: the same angles for every grain
    AmpPlan plan((int64_t)ang.size(), nmax_chunk);
    std::vector<AmpUse> uses;
    std::vector<TmxQJob> qj;
    const int64_t per_theta = 1 + (account ? (int64_t)ngauss * ngauss : 0);
    const int64_t sca_base = ng * ntheta * per_theta;
    std::vector<AmpJob> jobs;
    for (int t = 0; t < ntheta; ++t) {
      jobs.push_back({t, t, 1, 0, t * per_theta});
      for (int ti = 0; account && ti < ngauss; ++ti) {
        jobs.push_back({acc_a0 + ti, t, ngauss, acc_p0,
                        t * per_theta + 1 + (int64_t)ti * ngauss});
      }
    }
    const auto main_groups = plan.add(jobs);
    jobs.clear();
    for (int t = 0; do_sca && t < ntheta; ++t) {
      jobs.push_back({sca_ain, sca_a0 + t, nphi_sca, sca_p0, (int64_t)t * nphi_sca});
    }
    const auto sca_groups = plan.add(jobs);
    for (int64_t g = 0; g < ng; ++g) {
      if (og[g].nmax <= 0) {
        continue;
      }
      const int64_t out0 = g * ntheta * per_theta;
      uses.push_back({(int32_t)g, main_groups.first, main_groups.second, out0});
      uses.push_back({(int32_t)g, sca_groups.first, sca_groups.second,
                      sca_base + g * ntheta * nphi_sca});
      for (int t = 0; t < ntheta; ++t) {
        TmxQJob q;
        q.grain = (int32_t)g;
        q.pad = 0;
        q.out = g * ntheta + t;
        q.s_main = out0 + t * per_theta;
        q.s_acc = q.s_main + 1;
        qj.push_back(q);
      }
    }
    const int64_t nsca = do_sca ? ng * ntheta * nphi_sca : 0;
    const int64_t s_total = sca_base + nsca;
    if ((rc = ensure(ctx, ctx->o_qj, std::max<size_t>(1, qj.size()) * sizeof(TmxQJob))) ||
        (rc = ensure(ctx, ctx->o_S, std::max<int64_t>(1, s_total) * 4 * sizeof(cplx))) ||
        (rc = ensure(ctx, ctx->o_gq, std::max<int64_t>(1, ng * ntheta * nq) * sizeof(double))) ||
        (rc = ensure(ctx, ctx->o_gz, std::max<int64_t>(1, do_sca ? nsca * 16 : 1) * sizeof(double))) ||
        (rc = ensure(ctx, ctx->o_cq, std::max<int64_t>(1, nc * ntheta * nq) * sizeof(double))) ||
        (rc = ensure(ctx, ctx->o_cz, std::max<int64_t>(1, do_sca ? nc * ntheta * nphi_sca * 16 : 1) * sizeof(double)))) {
      return rc;
    }
    if (!qj.empty()) {
      CK(cudaMemcpyAsync(ctx->o_qj.p, qj.data(), qj.size() * sizeof(TmxQJob),
                         cudaMemcpyHostToDevice, st));
    }
    if ((rc = upload_obs_plan(ctx, og, ang, plan, std::move(uses))) ||
        (ctx->obs_s_valid = false, false) ||
        (rc = run_amplitudes(ctx, (const cplx *)ctx->T.p, t_total, ncoef,
                             (cplx *)ctx->o_S.p, s_total))) {
      return rc;
    }
    if (nq > 0) {
      CK(cudaMemsetAsync(ctx->o_gq.p, 0, ng * ntheta * nq * sizeof(double), st));
      tmx_launch_q_epilogue((const TmxQJob *)ctx->o_qj.p, (int)qj.size(),
                            (const TmxObsGrain *)ctx->o_og.p, (const cplx *)ctx->o_S.p,
                            (const double *)ctx->o_wts.p, account ? ngauss : 0,
                            (double *)ctx->o_gq.p, nq, do_abs, do_ext, st);
      LAUNCHED();
      cudaEvent_t pe = nullptr;
      if ((rc = prof_begin(ctx, TMX_PROF_SHAPE_AVG, &pe))) {
        return rc;
      }
      tmx_launch_shape_avg((int)nc, nshape, ntheta * nq, (const double *)ctx->o_gq.p,
                           (const double *)ctx->o_shw.p, (double *)ctx->o_cq.p, st);
      LAUNCHED();
      // per cell: nshape inputs and one output per coefficient, the weights
      if ((rc = prof_end(ctx, TMX_PROF_SHAPE_AVG, pe, 0., st,
                         8. * (nc * (nshape + 1.) * ntheta * nq + nshape)))) {
        return rc;
      }
      CK(cudaMemcpyAsync(out_q + c0 * ntheta * nq, ctx->o_cq.p,
                         nc * ntheta * nq * sizeof(double), cudaMemcpyDeviceToHost, st));
    }
    if (do_sca) {
      tmx_launch_z_epilogue((int)nsca, (const cplx *)ctx->o_S.p + sca_base * 4,
                            (double *)ctx->o_gz.p, st);
      LAUNCHED();
      cudaEvent_t pz = nullptr;
      if ((rc = prof_begin(ctx, TMX_PROF_SHAPE_AVG, &pz))) {
        return rc;
      }
      tmx_launch_shape_avg((int)nc, nshape, ntheta * nphi_sca * 16,
                           (const double *)ctx->o_gz.p, (const double *)ctx->o_shw.p,
                           (double *)ctx->o_cz.p, st);
      LAUNCHED();
      if ((rc = prof_end(ctx, TMX_PROF_SHAPE_AVG, pz, 0., st,
                         8. * (nc * (nshape + 1.) * ntheta * nphi_sca * 16 + nshape)))) {
        return rc;
      }
      CK(cudaMemcpyAsync(out_z + c0 * ntheta * nphi_sca * 16, ctx->o_cz.p,
                         nc * ntheta * nphi_sca * 16 * sizeof(double),
                         cudaMemcpyDeviceToHost, st));
    }
    CK(cudaStreamSynchronize(st));
    c0 = c1;
  }
  return TMX_OK;
}

// Clebsch-Gordan table for every (n1, n2) up to nmax (cached; rebuilt when a
// larger nmax is needed)
int tmx_ensure_cg(tmx_ctx *ctx, int nmax) {
  if (ctx->cg_nmax >= nmax && ctx->cg_nmax > 0) {
    return TMX_OK;
  }
  nmax = std::max(nmax, ctx->cg_nmax);
  cudaStream_t st = ctx->stream;
  std::vector<int64_t> off((size_t)nmax * nmax);
  int64_t tot = 0;
  for (int n1 = 1; n1 <= nmax; ++n1) {
    for (int n2 = 1; n2 <= nmax; ++n2) {
      const int M = std::min(n1, n2);
      off[(size_t)(n1 - 1) * nmax + (n2 - 1)] = tot;
      tot += (int64_t)(2 * M + 1) * (M + 1);
    }
  }
  // a thread per row of the table, as many as stay resident at most; each has two
  // rows of work space
  const int64_t rows = (int64_t)nmax * nmax * (2 * nmax + 1);
  const int blocks = (int)std::min<int64_t>(4 * 148, (rows + 127) / 128);
  int rc;
  if ((rc = ensure(ctx, ctx->cg, tot * sizeof(double))) ||
      (rc = ensure(ctx, ctx->cg_off, off.size() * sizeof(int64_t))) ||
      (rc = ensure(ctx, ctx->o_work,
                   (size_t)blocks * 128 * 2 * (2 * nmax + 1) * sizeof(double)))) {
    return rc;
  }
  CK(cudaMemcpyAsync(ctx->cg_off.p, off.data(), off.size() * sizeof(int64_t),
                     cudaMemcpyHostToDevice, st));
  tmx_launch_cg(nmax, (const int64_t *)ctx->cg_off.p, (double *)ctx->cg.p,
                (double *)ctx->o_work.p, blocks, st);
  LAUNCHED();
  CK(cudaStreamSynchronize(st));
  ctx->cg_nmax = nmax;
  return TMX_OK;
}

// ------------------------------------------- per-grain observables / grads --

namespace {

// orientation-averaged theta -> theta amplitudes of every grain of the last
// batch for the T-matrices at `Tsrc`; S[(grain * ntheta + t) * 4]
int batch_amplitudes(tmx_ctx *ctx, const cplx *Tsrc, int ntheta, int ncoef,
                     cplx *S_out) {
  return run_amplitudes(ctx, Tsrc, ctx->p2_t_total, ncoef, S_out,
                        ctx->n * ntheta);
}

// descriptors shared by the per-grain observable and gradient passes
int batch_observable_setup(tmx_ctx *ctx, int ntheta, const double *thetas,
                           const double *coeffs, int ncoef) {
  cudaStream_t st = ctx->stream;
  const int64_t n = ctx->n;
  int rc;
  // the plan of the previous call, if nothing it depends on has changed
  // since (the observables of a batch followed by its gradients)
  tmx_ctx::ObsKey &key = ctx->obs_key;
  if (key.valid && key.batch_seq == ctx->batch_seq && key.plan_seq == ctx->plan_seq &&
      key.has_coeffs == (coeffs != nullptr) && (int)key.thetas.size() == ntheta &&
      std::equal(key.thetas.begin(), key.thetas.end(), thetas) &&
      (!coeffs || ((int)key.coeffs.size() == ncoef &&
                   std::equal(key.coeffs.begin(), key.coeffs.end(), coeffs)))) {
    return TMX_OK;
  }
  key.valid = false;
  ctx->obs_s_valid = false;
  std::vector<TmxAngle> ang(ntheta);
  for (int i = 0; i < ntheta; ++i) {
    ang[i] = make_angle(cos(thetas[i]));
  }
  std::vector<cplx> phis(1, mkc(1., 0.));
  std::vector<TmxObsGrain> og(n);
  int nmax_b = 1;
  for (int64_t g = 0; g < n; ++g) {
    nmax_b = std::max(nmax_b, ctx->nmax_h[g]);
  }
  AmpPlan plan(ntheta, nmax_b);
  std::vector<AmpJob> jobs;
  for (int t = 0; t < ntheta; ++t) {
    jobs.push_back({t, t, 1, 0, t});
  }
  const auto groups = plan.add(jobs);
  std::vector<AmpUse> uses;
  std::vector<TmxQJob> qj;
  qj.reserve((size_t)n * ntheta);
  for (int64_t g = 0; g < n; ++g) {
    og[g].nmax = ctx->nmax_h[g];
    og[g].coef_set = coeffs ? 0 : -1;
    og[g].t_off = ctx->t_off_h[g];
    og[g].k = ctx->up_grains[g].k;
    og[g].r_ev = ctx->up_grains[g].r_ev;
    if (coeffs && 2 * og[g].nmax + 1 > ncoef) {
      return fail(ctx, TMX_ERR_INVALID,
                  "orientation coefficients shorter than 2 nmax + 1");
    }
    if (og[g].nmax <= 0) {
      continue;
    }
    uses.push_back({(int32_t)g, groups.first, groups.second, g * ntheta});
    for (int t = 0; t < ntheta; ++t) {
      TmxQJob q;
      q.grain = (int32_t)g;
      q.pad = 0;
      q.out = g * ntheta + t;
      q.s_main = g * ntheta + t;
      q.s_acc = 0;
      qj.push_back(q);
    }
  }
  if ((rc = ensure(ctx, ctx->o_phis, sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->o_og, std::max<int64_t>(1, n) * sizeof(TmxObsGrain))) ||
      (rc = ensure(ctx, ctx->o_qj, std::max<size_t>(1, qj.size()) * sizeof(TmxQJob))) ||
      (rc = ensure(ctx, ctx->o_coef, std::max(1, ncoef) * sizeof(double)))) {
    return rc;
  }
  CK(cudaMemcpyAsync(ctx->o_phis.p, phis.data(), sizeof(cplx),
                     cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(ctx->o_og.p, og.data(), n * sizeof(TmxObsGrain),
                     cudaMemcpyHostToDevice, st));
  if (!qj.empty()) {
    CK(cudaMemcpyAsync(ctx->o_qj.p, qj.data(), qj.size() * sizeof(TmxQJob),
                       cudaMemcpyHostToDevice, st));
  }
  if (coeffs) {
    CK(cudaMemcpyAsync(ctx->o_coef.p, coeffs, ncoef * sizeof(double),
                       cudaMemcpyHostToDevice, st));
  }
  ctx->o_nqj = (int)qj.size();
  if (coeffs && (rc = tmx_ensure_cg(ctx, nmax_b))) {
    return rc;
  }
  if ((rc = upload_obs_plan(ctx, og, ang, plan, std::move(uses)))) {
    return rc;
  }
  key.valid = true;
  key.batch_seq = ctx->batch_seq;
  key.plan_seq = ctx->plan_seq;
  key.thetas.assign(thetas, thetas + ntheta);
  key.has_coeffs = coeffs != nullptr;
  if (coeffs) {
    key.coeffs.assign(coeffs, coeffs + ncoef);
  } else {
    key.coeffs.clear();
  }
  return TMX_OK;
}

} // namespace

extern "C" int tmx_batch_observables(tmx_ctx *ctx, int32_t ntheta,
                                     const double *thetas, const double *coeffs,
                                     int32_t ncoef, double *q) {
  if (!ctx || ntheta < 1 || !thetas || !q) {
    return TMX_ERR_INVALID;
  }
  if (!ctx->have_batch) {
    return fail(ctx, TMX_ERR_STATE, "no batch has been computed");
  }
  CK(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const int64_t n = ctx->n;
  int rc;
  if ((rc = batch_observable_setup(ctx, ntheta, thetas, coeffs, ncoef)) ||
      (rc = ensure(ctx, ctx->o_S, std::max<int64_t>(1, n * ntheta) * 4 * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->o_gq, std::max<int64_t>(1, n * ntheta * 3) * sizeof(double)))) {
    return rc;
  }
  ctx->obs_s_valid = false;
  if ((rc = batch_amplitudes(ctx, (const cplx *)ctx->T.p, ntheta, ncoef,
                             (cplx *)ctx->o_S.p))) {
    return rc;
  }
  ctx->obs_s_valid = true;
  CK(cudaMemsetAsync(ctx->o_gq.p, 0, n * ntheta * 3 * sizeof(double), st));
  tmx_launch_q_epilogue((const TmxQJob *)ctx->o_qj.p, ctx->o_nqj,
                        (const TmxObsGrain *)ctx->o_og.p, (const cplx *)ctx->o_S.p,
                        nullptr, 0, (double *)ctx->o_gq.p, 3, 0, 1, st);
  LAUNCHED();
  CK(cudaMemcpyAsync(q, ctx->o_gq.p, n * ntheta * 3 * sizeof(double),
                     cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return TMX_OK;
}

extern "C" int tmx_batch_gradients(tmx_ctx *ctx, int32_t ntheta,
                                   const double *thetas, const double *coeffs,
                                   int32_t ncoef, double *q, double *dq) {
  if (!ctx || ntheta < 1 || !thetas || !dq) {
    return TMX_ERR_INVALID;
  }
  if (!ctx->have_batch) {
    return fail(ctx, TMX_ERR_STATE, "no batch has been computed");
  }
  CK(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const int64_t n = ctx->n;
  int rc;
  if (ctx->t_averaged) {
    return fail(ctx, TMX_ERR_STATE,
                "gradients need the batch's own T-matrices, not orientation averages");
  }
  // LU factors of every item: kept by the batch's block rounds, or by a
  // single-round batch in the p2 set; otherwise the forward blocks run again
  // in one round that keeps them
  if (!ctx->rounds_lu && ctx->p2_rounds > 1 && (rc = tmx_rerun_blocks(ctx))) {
    return rc;
  }
  struct RoundView {
    const TmxItem *items;
    const TmxSlot *slots;
    const double *tab, *nsc;
    cplx *lu;
    std::vector<std::array<int64_t, 3>> seg; // size buckets: [i0, i1), max class size
    int64_t scr;
  };
  // the class-size buckets of a round whose items are sorted by size,
  // largest first
  auto segments = [](const std::vector<int> &nb) {
    std::vector<std::array<int64_t, 3>> seg;
    const int edges[] = {1 << 30, 64, 32, 16, 8, 0};
    const int64_t nitems = (int64_t)nb.size();
    int64_t i0 = 0;
    for (int b = 0; b < 5; ++b) {
      int64_t i1 = i0;
      int mx = 0;
      while (i1 < nitems && nb[i1] > edges[b + 1]) {
        mx = std::max(mx, nb[i1]);
        ++i1;
      }
      if (i1 > i0) {
        seg.push_back({i0, i1, (int64_t)mx});
      }
      i0 = i1;
    }
    return seg;
  };
  std::vector<RoundView> views;
  // scratch of a round's tangents: only the classes above 32 members keep dQ
  // and dRgQ in memory (tmx_launch_tangents). Rounds made by the host lay the
  // items' scratch out largest first, so theirs is the front of it; a round
  // made on the device mixes the sizes.
  auto large_scratch = [](const std::vector<int> &nb) {
    int64_t s = 0;
    for (size_t i = 0; i < nb.size() && nb[i] > 32; ++i) {
      s += tmx_item_scratch(nb[i]);
    }
    return s;
  };
  if (ctx->rounds_lu) {
    for (const auto &r : ctx->rounds_kept) {
      const bool host = r.seg.empty();
      const auto seg = host ? segments(r.nb) : r.seg;
      const bool large = !seg.empty() && seg[0][2] > 32;
      views.push_back({r.items, r.slots, r.tab, r.nsc, r.lu, seg,
                       host ? large_scratch(r.nb) : large ? r.scr_total : 0});
    }
  } else {
    if ((rc = ensure(ctx, ctx->lu, std::max<int64_t>(1, ctx->p2_scr_total) * sizeof(cplx)))) {
      return rc;
    }
    views.push_back({(const TmxItem *)ctx->p2items.p, (const TmxSlot *)ctx->p2slots.p,
                     (const double *)ctx->p2tab.p, (const double *)ctx->p2nsc.p,
                     (cplx *)ctx->lu.p, segments(ctx->p2_nb),
                     large_scratch(ctx->p2_nb)});
  }
  // each round's tangent scratch in its own region: the rounds' size
  // buckets run concurrently
  int64_t scr_sum = 1;
  for (const RoundView &v : views) {
    scr_sum += v.scr;
  }
  const int64_t tt = ctx->p2_t_total;
  NvtxRange range("tmx_gradients");
  if ((rc = ensure(ctx, ctx->tscr, 3 * scr_sum * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->dT, std::max<int64_t>(1, 3 * tt) * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->dS, std::max<int64_t>(1, 4 * n * ntheta) * 4 * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->o_gq, std::max<int64_t>(1, n * ntheta * 3) * sizeof(double))) ||
      (rc = ensure(ctx, ctx->o_gz, std::max<int64_t>(1, n * ntheta * 12) * sizeof(double)))) {
    return rc;
  }
  CK(cudaMemsetAsync(ctx->dT.p, 0, std::max<int64_t>(1, 3 * tt) * sizeof(cplx), st));
  // every (round, size bucket) launch may start once dT is cleared: they
  // write disjoint blocks of dT and disjoint scratch, so they run on the
  // library stream and the eight others side by side and join before the
  // observables
  cudaStream_t gstreams[9] = {st,          ctx->aux[0], ctx->aux[1],
                              ctx->aux[2], ctx->aux[3], ctx->aux[4],
                              ctx->aux[5], ctx->stream2, ctx->stream3};
  cudaEvent_t gfork;
  CK(cudaEventCreateWithFlags(&gfork, cudaEventDisableTiming));
  CK(cudaEventRecord(gfork, st));
  bool gused[9] = {true, false, false, false, false, false, false, false, false};
  int glaunch = 0;
  int64_t scr_off = 0;
  for (const RoundView &v : views) {
    for (const auto &sg : v.seg) {
      const int64_t i0 = sg[0], i1 = sg[1];
      const int max_nb = (int)sg[2];
      {
        const int gi = glaunch++ % 9;
        cudaStream_t gs = gstreams[gi];
        if (!gused[gi]) {
          CK(cudaStreamWaitEvent(gs, gfork, 0));
          gused[gi] = true;
        }
        if (!ctx->rounds_lu && !ctx->lu_ready) {
          TmxBlockArgs B;
          B.items = v.items + i0;
          B.nitems = (int)(i1 - i0);
          B.slots = v.slots;
          B.grains = (const TmxGrain *)ctx->grains.p;
          B.tab = v.tab;
          B.nsc = v.nsc;
          B.wig = (const double *)ctx->wig.p;
          B.wig_off = (const int64_t *)ctx->wig_off.p;
          B.scratch = (cplx *)ctx->p2scratch.p;
          B.tout = (cplx *)ctx->T.p;
          B.diag = nullptr;
          B.status = (int32_t *)ctx->status.p;
          B.max_nb = max_nb;
          B.family = dispatch_family(ctx, max_nb);
          B.lu = v.lu;
          LAUNCHED_N(tmx_launch_blocks(B, gs));
        }
        TmxTangentArgs A;
        A.items = v.items + i0;
        A.nitems = (int)(i1 - i0);
        A.nparams = 3;
        A.slots = v.slots;
        A.grains = (const TmxGrain *)ctx->grains.p;
        A.tab = v.tab;
        A.nsc = v.nsc;
        A.wig = (const double *)ctx->wig.p;
        A.wig_off = (const int64_t *)ctx->wig_off.p;
        A.lu = v.lu;
        A.T = (const cplx *)ctx->T.p;
        A.scratch = (cplx *)ctx->tscr.p + 3 * scr_off;
        A.scratch_stride = v.scr;
        A.dT = (cplx *)ctx->dT.p;
        A.dT_stride = tt;
        A.chunk_nodes = std::max(1, tmx_host_chunk_nodes(max_nb) / 2);
        A.max_nb = max_nb;
        cudaEvent_t pe = nullptr;
        if ((rc = prof_begin(ctx, TMX_PROF_TANGENTS, &pe, gs))) {
          return rc;
        }
        tmx_launch_tangents(A, gs);
        LAUNCHED();
        if ((rc = prof_end(ctx, TMX_PROF_TANGENTS, pe, 0., gs, 0., A.nitems))) {
          return rc;
        }
      }
    }
    scr_off += v.scr;
  }
  for (int gi = 1; gi < 9; ++gi) {
    if (gused[gi]) {
      CK(cudaEventRecord(gfork, gstreams[gi]));
      CK(cudaStreamWaitEvent(st, gfork, 0));
    }
  }
  CK(cudaEventDestroy(gfork));
  if ((rc = batch_observable_setup(ctx, ntheta, thetas, coeffs, ncoef))) {
    return rc;
  }
  cplx *S = (cplx *)ctx->dS.p;
  const int64_t sz = n * ntheta * 4;
  // the T-matrices' own amplitudes: those of tmx_batch_observables when it
  // ran on this batch with the same plan (still in o_S), else computed here
  const bool have_s = ctx->obs_s_valid;
  const cplx *S0 = have_s ? (const cplx *)ctx->o_S.p : S;
  {
    // the three tangents (and T) in one pass (shared angle and coupling work)
    const cplx *src[4] = {(const cplx *)ctx->T.p, (const cplx *)ctx->dT.p,
                          (const cplx *)ctx->dT.p + tt, (const cplx *)ctx->dT.p + 2 * tt};
    cplx *dst[4] = {S, S + sz, S + 2 * sz, S + 3 * sz};
    const int k0 = have_s ? 1 : 0;
    if ((rc = run_amplitudes(ctx, src + k0, 4 - k0, ctx->p2_t_total, ncoef, dst + k0,
                             n * ntheta))) {
      return rc;
    }
  }
  CK(cudaMemsetAsync(ctx->o_gq.p, 0, n * ntheta * 3 * sizeof(double), st));
  CK(cudaMemsetAsync(ctx->o_gz.p, 0, n * ntheta * 12 * sizeof(double), st));
  tmx_launch_q_epilogue((const TmxQJob *)ctx->o_qj.p, ctx->o_nqj,
                        (const TmxObsGrain *)ctx->o_og.p, S0, nullptr, 0,
                        (double *)ctx->o_gq.p, 3, 0, 1, st);
  LAUNCHED();
  tmx_launch_dq_epilogue((const TmxQJob *)ctx->o_qj.p, ctx->o_nqj,
                         (const TmxObsGrain *)ctx->o_og.p, S0, S + sz, S + 2 * sz,
                         S + 3 * sz, (double *)ctx->o_gz.p, st);
  LAUNCHED();
  if (q) {
    CK(cudaMemcpyAsync(q, ctx->o_gq.p, n * ntheta * 3 * sizeof(double),
                       cudaMemcpyDeviceToHost, st));
  }
  CK(cudaMemcpyAsync(dq, ctx->o_gz.p, n * ntheta * 12 * sizeof(double),
                     cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return TMX_OK;
}

// ------------------------------------------ plain-path observables (A25) --

namespace {

// Lab-frame direction (theta, phi) in the frame of a particle whose symmetry
// axis points at (beta, alpha), and the 2 x 2 amplitude rotation between the
// frames (TMatrix::get_forward_scattering_matrix, TMatrix.hpp:1306-1420).
struct PDir {
  TmxAngle a;        // cos, sin, 1/sin (or 9000) of the particle zenith
  double cphi, sphi; // particle azimuth
  double R[2][2];    // AP B AL
};

PDir particle_dir(double cosalpha, double sinalpha, double cosbeta,
                  double sinbeta, double theta, double phi) {
  PDir d;
  const double ct = cos(theta), st = sin(theta);
  const double cp = cos(phi), sp = sin(phi);
  const double cosphirel = cp * cosalpha + sp * sinalpha;
  const double sinphirel = sp * cosalpha - cp * sinalpha;
  const double ctp = ct * cosbeta + st * sinbeta * cosphirel;
  const double stp = sin(acos(ctp));
  double cphi, sphi, sinv;
  if (stp != 0.) {
    sinv = 1. / stp;
    cphi = (cosbeta * st * cosphirel - sinbeta * ct) * sinv;
    sphi = st * sinphirel * sinv;
  } else {
    cphi = 1.;
    sphi = 0.;
    sinv = 9000.;
  }
  d.a.c = ctp;
  d.a.s = stp;
  d.a.si = sinv;
  d.cphi = cphi;
  d.sphi = sphi;
  const double B[3][3] = {{cosalpha * cosbeta, sinalpha * cosbeta, -sinbeta},
                          {-sinalpha, cosalpha, 0.},
                          {cosalpha * sinbeta, sinalpha * sinbeta, cosbeta}};
  const double AL[3][2] = {{ct * cp, -sp}, {ct * sp, cp}, {-st, 0.}};
  const double AP[2][3] = {{ctp * cphi, ctp * sphi, -stp}, {-sphi, cphi, 0.}};
  double C[3][2];
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 2; ++j) {
      C[i][j] = 0.;
      for (int k = 0; k < 3; ++k) {
        C[i][j] += B[i][k] * AL[k][j];
      }
    }
  }
  for (int i = 0; i < 2; ++i) {
    for (int j = 0; j < 2; ++j) {
      d.R[i][j] = 0.;
      for (int k = 0; k < 3; ++k) {
        d.R[i][j] += AP[i][k] * C[k][j];
      }
    }
  }
  return d;
}

// direction of a particle-frame zenith angle without rotation (the
// four-angle form of get_forward_scattering_matrix, TMatrix.hpp:1245-1290)
TmxAngle plain_angle(double theta) {
  TmxAngle a;
  a.c = cos(theta);
  a.s = sin(theta);
  a.si = (a.s != 0.) ? 1. / a.s : 9000.;
  return a;
}

typedef std::complex<double> zc;

// Z from the 2 x 2 amplitude matrix S (TMatrix.hpp:1896-1948), row major
void z_from_s(const zc S[2][2], double *Z) {
  const zc ic(0., 1.);
  const double half(0.5);
  Z[0] = (half * (S[0][0] * conj(S[0][0]) + S[0][1] * conj(S[0][1]) +
                  S[1][0] * conj(S[1][0]) + S[1][1] * conj(S[1][1])))
             .real();
  Z[1] = (half * (S[0][0] * conj(S[0][0]) - S[0][1] * conj(S[0][1]) +
                  S[1][0] * conj(S[1][0]) - S[1][1] * conj(S[1][1])))
             .real();
  Z[2] = (-S[0][0] * conj(S[0][1]) - S[1][1] * conj(S[1][0])).real();
  Z[3] = (ic * (S[0][0] * conj(S[0][1]) - S[1][1] * conj(S[1][0]))).real();
  Z[4] = (half * (S[0][0] * conj(S[0][0]) + S[0][1] * conj(S[0][1]) -
                  S[1][0] * conj(S[1][0]) - S[1][1] * conj(S[1][1])))
             .real();
  Z[5] = (half * (S[0][0] * conj(S[0][0]) - S[0][1] * conj(S[0][1]) -
                  S[1][0] * conj(S[1][0]) + S[1][1] * conj(S[1][1])))
             .real();
  Z[6] = (-S[0][0] * conj(S[0][1]) + S[1][1] * conj(S[1][0])).real();
  Z[7] = (ic * (S[0][0] * conj(S[0][1]) + S[1][1] * conj(S[1][0]))).real();
  Z[8] = (-S[0][0] * conj(S[1][0]) - S[1][1] * conj(S[0][1])).real();
  Z[9] = (-S[0][0] * conj(S[1][0]) + S[1][1] * conj(S[0][1])).real();
  Z[10] = (S[0][0] * conj(S[1][1]) + S[0][1] * conj(S[1][0])).real();
  Z[11] = (-ic * (S[0][0] * conj(S[1][1]) + S[1][0] * conj(S[0][1]))).real();
  Z[12] = (ic * (S[1][0] * conj(S[0][0]) + S[1][1] * conj(S[0][1]))).real();
  Z[13] = (ic * (S[1][0] * conj(S[0][0]) - S[1][1] * conj(S[0][1]))).real();
  Z[14] = (-ic * (S[1][1] * conj(S[0][0]) - S[0][1] * conj(S[1][0]))).real();
  Z[15] = (S[1][1] * conj(S[0][0]) - S[0][1] * conj(S[1][0])).real();
}

// K from the forward amplitude matrix (TMatrix.hpp:1972-2010), row major
void k_from_s(double k, const zc S[2][2], double *K) {
  const double pf = 2. * M_PI / k;
  for (int i = 0; i < 16; ++i) {
    K[i] = 0.;
  }
  K[0] = pf * (S[0][0] + S[1][1]).imag();
  K[5] = K[0];
  K[10] = K[0];
  K[15] = K[0];
  K[1] = pf * (S[0][0] - S[1][1]).imag();
  K[4] = K[1];
  K[2] = -pf * (S[0][1] + S[1][0]).imag();
  K[8] = K[2];
  K[3] = pf * (S[1][0] - S[0][1]).real();
  K[12] = K[3];
  K[6] = pf * (S[1][0] - S[0][1]).imag();
  K[9] = -K[6];
  K[7] = -pf * (S[0][1] + S[1][0]).real();
  K[13] = -K[7];
  K[11] = pf * (S[1][1] - S[0][0]).real();
  K[14] = -K[11];
}

// Amplitude matrices S^P of nj jobs (the j-th for grain(j): incoming and
// outgoing angle, azimuths e^{i(phi_out - phi_in)}) for the T-matrices of the
// last batch (plain or averaged); ns amplitudes in all, at the jobs' places.
template <class Grain, class Job>
int plain_amplitudes(tmx_ctx *ctx, int64_t nj, Grain grain, Job job,
                     const std::vector<TmxAngle> &ang, const std::vector<cplx> &e1,
                     int64_t ns, std::vector<zc> &S) {
  cudaStream_t st = ctx->stream;
  const int64_t n = ctx->n;
  int rc;
  std::vector<TmxObsGrain> og(n);
  int nbmax = 1;
  for (int64_t g = 0; g < n; ++g) {
    og[g].nmax = ctx->nmax_h[g];
    og[g].coef_set = -1;
    og[g].t_off = ctx->t_off_h[g];
    og[g].k = ctx->up_grains[g].k;
    og[g].r_ev = ctx->up_grains[g].r_ev;
    nbmax = std::max(nbmax, og[g].nmax);
  }
  if ((rc = ensure(ctx, ctx->o_og, std::max<int64_t>(1, n) * sizeof(TmxObsGrain))) ||
      (rc = ensure(ctx, ctx->o_phis, std::max<size_t>(1, e1.size()) * sizeof(cplx))) ||
      (rc = ensure(ctx, ctx->o_S, std::max<int64_t>(1, ns) * 4 * sizeof(cplx)))) {
    return rc;
  }
  // jobs by grain (a stable counting sort), those of grains without a T left out
  std::vector<int32_t> start(n + 1, 0);
  for (int64_t j = 0; j < nj; ++j) {
    start[grain(j) + 1] += og[grain(j)].nmax > 0 ? 1 : 0;
  }
  for (int64_t g = 0; g < n; ++g) {
    start[g + 1] += start[g];
  }
  std::vector<int32_t> by(start[n]);
  std::vector<int32_t> pos(start.begin(), start.end() - 1);
  for (int64_t j = 0; j < nj; ++j) {
    if (og[grain(j)].nmax > 0) {
      by[pos[grain(j)]++] = (int32_t)j;
    }
  }
  AmpPlan plan((int64_t)ang.size(), nbmax);
  std::vector<AmpUse> uses;
  for (int64_t g = 0; g < n; ++g) {
    if (start[g + 1] > start[g]) {
      const int32_t *own = by.data() + start[g];
      const auto gr = plan.add(start[g + 1] - start[g],
                               [&](int32_t j) { return job(own[j]); });
      uses.push_back({(int32_t)g, gr.first, gr.second, 0});
    }
  }
  ++ctx->plan_seq; // the observable buffers change below
  ctx->obs_s_valid = false;
  CK(cudaMemcpyAsync(ctx->o_og.p, og.data(), n * sizeof(TmxObsGrain),
                     cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(ctx->o_phis.p, e1.data(), e1.size() * sizeof(cplx),
                     cudaMemcpyHostToDevice, st));
  if ((rc = upload_obs_plan(ctx, og, ang, plan, std::move(uses))) ||
      (rc = run_amplitudes(ctx, (const cplx *)ctx->T.p, ctx->p2_t_total, 1,
                           (cplx *)ctx->o_S.p, ns))) {
    return rc;
  }
  static_assert(sizeof(zc) == sizeof(cplx), "both are (re, im) in doubles");
  S.resize(4 * ns);
  CK(cudaMemcpyAsync(S.data(), ctx->o_S.p, 4 * ns * sizeof(cplx), cudaMemcpyDeviceToHost,
                     st));
  CK(cudaStreamSynchronize(st));
  return TMX_OK;
}

int check_jobs(tmx_ctx *ctx, int64_t njobs, const int64_t *grain) {
  if (!ctx->have_batch) {
    return fail(ctx, TMX_ERR_STATE, "no batch has been computed");
  }
  for (int64_t j = 0; j < njobs; ++j) {
    if (grain[j] < 0 || grain[j] >= ctx->n) {
      return fail(ctx, TMX_ERR_INVALID, "grain index out of range");
    }
  }
  return TMX_OK;
}

// lab-frame S for jobs at particle orientations: S^L = R_out^-1 S^P R_in
// (TMatrix.hpp:1420-1460)
int lab_amplitudes(tmx_ctx *ctx, int64_t njobs, const int64_t *grain,
                   const double *alpha, const double *beta,
                   const double *theta_in, const double *phi_in,
                   const double *theta_out, const double *phi_out,
                   std::vector<zc> &SL) {
  std::vector<std::array<int32_t, 2>> pair(njobs); // angles in, out
  std::vector<cplx> e1(njobs);
  struct Rot {
    double in[2][2], out[2][2];
  };
  std::vector<Rot> rot(njobs);
  // Particle-frame zeniths that repeat get one number. The numbers seen last
  // are kept in pairs by hash, in a table that stays in the cache: an angle
  // pushed out of it gets a second number, which costs its columns again but
  // nothing else (100,000 jobs with directions of their own: 7 ms in one hash
  // table of all angles, 2.5 ms in this one).
  std::vector<TmxAngle> ang;
  ang.reserve(2 * (size_t)njobs);
  struct Seen {
    uint32_t tag[2];
    int32_t number[2];
  };
  size_t places = 16;
  while (places < (size_t)njobs && places < 32768) {
    places *= 2;
  }
  std::vector<Seen> seen(places, Seen{{0, 0}, {-1, -1}});
  const auto angle = [&](const TmxAngle &a) {
    uint64_t h[3];
    memcpy(h, &a, sizeof(h));
    // (cos, sin) name the angle; 1 / sin follows from sin
    const uint64_t key = (h[0] ^ (h[1] >> 1)) * 0x9E3779B97F4A7C15ull;
    const uint32_t tag = (uint32_t)(key >> 32);
    Seen &e = seen[(key >> 16) & (places - 1)];
    for (int w = 0; w < 2; ++w) {
      const int32_t i = e.number[w];
      if (e.tag[w] == tag && i >= 0 && memcmp(&ang[i], &a, sizeof(a)) == 0) {
        return i;
      }
    }
    e.tag[1] = e.tag[0];
    e.number[1] = e.number[0];
    e.tag[0] = tag;
    e.number[0] = (int32_t)ang.size();
    ang.push_back(a);
    return e.number[0];
  };
  for (int64_t j = 0; j < njobs; ++j) {
    const double ca = cos(alpha[j]), sa = sin(alpha[j]);
    const double cb = cos(beta[j]), sb = sin(beta[j]);
    const PDir din = particle_dir(ca, sa, cb, sb, theta_in[j], phi_in[j]);
    const PDir dout = particle_dir(ca, sa, cb, sb, theta_out[j], phi_out[j]);
    pair[j] = {angle(din.a), angle(dout.a)};
    e1[j] = mkc(dout.cphi * din.cphi + dout.sphi * din.sphi,
                dout.sphi * din.cphi - dout.cphi * din.sphi);
    memcpy(rot[j].in, din.R, sizeof(din.R));
    memcpy(rot[j].out, dout.R, sizeof(dout.R));
  }
  int rc = plain_amplitudes(
      ctx, njobs, [&](int64_t j) { return grain[j]; },
      [&](int64_t j) { return AmpJob{pair[j][0], pair[j][1], 1, j, j}; }, ang, e1, njobs, SL);
  if (rc) {
    return rc;
  }
  for (int64_t j = 0; j < njobs; ++j) {
    const zc S[4] = {SL[4 * j], SL[4 * j + 1], SL[4 * j + 2], SL[4 * j + 3]};
    const double(&Ri)[2][2] = rot[j].in;
    const double(&Rd)[2][2] = rot[j].out;
    double Ro[2][2];
    const double det = 1. / (Rd[0][0] * Rd[1][1] - Rd[0][1] * Rd[1][0]);
    Ro[0][0] = Rd[1][1] * det;
    Ro[0][1] = -Rd[0][1] * det;
    Ro[1][0] = -Rd[1][0] * det;
    Ro[1][1] = Rd[0][0] * det;
    const zc cS11 = S[0] * Ri[0][0] + S[1] * Ri[1][0];
    const zc cS12 = S[0] * Ri[0][1] + S[1] * Ri[1][1];
    const zc cS21 = S[2] * Ri[0][0] + S[3] * Ri[1][0];
    const zc cS22 = S[2] * Ri[0][1] + S[3] * Ri[1][1];
    SL[4 * j + 0] = Ro[0][0] * cS11 + Ro[0][1] * cS21;
    SL[4 * j + 1] = Ro[0][0] * cS12 + Ro[0][1] * cS22;
    SL[4 * j + 2] = Ro[1][0] * cS11 + Ro[1][1] * cS21;
    SL[4 * j + 3] = Ro[1][0] * cS12 + Ro[1][1] * cS22;
  }
  return TMX_OK;
}

// absorption cross sections (Cabs, Cabspol) of one grain at zenith angles
// th: per angle the forward amplitude and ngauss^2 incoming directions
// (TMatrix.hpp:2133-2200)
int absorption(tmx_ctx *ctx, int32_t grain, int32_t ntheta, const double *th,
               int32_t ngauss, double *out) {
  std::vector<double> ct(ngauss), wt(ngauss), ph(ngauss), wp(ngauss), tg(ngauss);
  tmx_host_gauss_legendre(ngauss, ct.data(), wt.data());
  gl_ab(ngauss, 0., 2. * M_PI, ph.data(), wp.data());
  for (int i = 0; i < ngauss; ++i) {
    tg[i] = acos(ct[i]);
  }
  std::vector<TmxAngle> ang;
  for (int i = 0; i < ngauss; ++i) {
    ang.push_back(plain_angle(tg[i]));
  }
  const int a0 = (int)ang.size();
  for (int t = 0; t < ntheta; ++t) {
    ang.push_back(plain_angle(th[t]));
  }
  // per angle the forward amplitude, then every incoming zenith with its
  // ngauss azimuths: e^{i(0 - phi_in)} as the reference forms it
  std::vector<AmpJob> jobs;
  std::vector<cplx> e1(1, mkc(1., 0.));
  for (int ip = 0; ip < ngauss; ++ip) {
    const double cp = cos(ph[ip]), sp = sin(ph[ip]);
    e1.push_back(mkc(1. * cp + 0. * sp, 0. * cp - 1. * sp));
  }
  int64_t ns = 0;
  for (int t = 0; t < ntheta; ++t) {
    jobs.push_back({a0 + t, a0 + t, 1, 0, ns++});
    for (int it = 0; it < ngauss; ++it) {
      jobs.push_back({it, a0 + t, ngauss, 1, ns});
      ns += ngauss;
    }
  }
  std::vector<zc> S;
  int rc = plain_amplitudes(
      ctx, (int64_t)jobs.size(), [&](int64_t) { return grain; },
      [&](int64_t j) { return jobs[j]; }, ang, e1, ns, S);
  if (rc) {
    return rc;
  }
  const double pf = 2. * M_PI / ctx->up_grains[grain].k;
  const double half(0.5);
  int64_t j = 0;
  for (int t = 0; t < ntheta; ++t) {
    const zc *s = S.data() + 4 * j++;
    double c0 = pf * (s[0] + s[3]).imag();
    double c1 = pf * (s[0] - s[3]).imag();
    for (int it = 0; it < ngauss; ++it) {
      for (int ip = 0; ip < ngauss; ++ip) {
        const zc *q = S.data() + 4 * j++;
        const double w = wt[it] * wp[ip];
        const double z00 = (half * (q[0] * conj(q[0]) + q[1] * conj(q[1]) +
                                    q[2] * conj(q[2]) + q[3] * conj(q[3])))
                               .real();
        const double z10 = (half * (q[0] * conj(q[0]) + q[1] * conj(q[1]) -
                                    q[2] * conj(q[2]) - q[3] * conj(q[3])))
                               .real();
        c0 -= z00 * w;
        c1 -= z10 * w;
      }
    }
    out[2 * t] = c0;
    out[2 * t + 1] = c1;
  }
  return TMX_OK;
}

} // namespace

extern "C" int tmx_batch_orientation_average(tmx_ctx *ctx, const double *coeffs,
                                             int32_t nsets, int32_t ncoef,
                                             const int32_t *coef_set) {
  if (!ctx || nsets < 0 || (nsets > 0 && (!coeffs || ncoef < 1))) {
    return TMX_ERR_INVALID;
  }
  if (!ctx->have_batch) {
    return fail(ctx, TMX_ERR_STATE, "no batch has been computed");
  }
  CK(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const int64_t n = ctx->n;
  int rc;
  std::vector<TmxObsGrain> og(n);
  int nmax_b = 1;
  for (int64_t g = 0; g < n; ++g) {
    og[g].nmax = ctx->nmax_h[g];
    og[g].coef_set = coef_set ? coef_set[g] : -1;
    og[g].t_off = ctx->t_off_h[g];
    og[g].k = ctx->up_grains[g].k;
    og[g].r_ev = ctx->up_grains[g].r_ev;
    if (og[g].coef_set >= nsets) {
      return fail(ctx, TMX_ERR_INVALID, "orientation set index");
    }
    if (og[g].coef_set >= 0 && og[g].nmax > 0 && 2 * og[g].nmax + 1 > ncoef) {
      return fail(ctx, TMX_ERR_INVALID,
                  "orientation coefficients shorter than 2 nmax + 1");
    }
    nmax_b = std::max(nmax_b, og[g].nmax);
  }
  const int64_t t_total = ctx->p2_t_total;
  if ((rc = ensure(ctx, ctx->o_og, std::max<int64_t>(1, n) * sizeof(TmxObsGrain))) ||
      (rc = ensure(ctx, ctx->o_coef, std::max<int64_t>(1, (int64_t)nsets * ncoef) * sizeof(double))) ||
      (rc = ensure(ctx, ctx->Ta, std::max<int64_t>(1, t_total) * sizeof(cplx))) ||
      (rc = tmx_ensure_cg(ctx, nmax_b))) {
    return rc;
  }
  ++ctx->plan_seq; // the observable buffers change below
  CK(cudaMemcpyAsync(ctx->o_og.p, og.data(), n * sizeof(TmxObsGrain),
                     cudaMemcpyHostToDevice, st));
  if (nsets > 0) {
    CK(cudaMemcpyAsync(ctx->o_coef.p, coeffs, (int64_t)nsets * ncoef * sizeof(double),
                       cudaMemcpyHostToDevice, st));
  }
  if ((rc = upload_obs_plan(ctx, og, {}, AmpPlan(0, 1), {}))) {
    return rc;
  }
  if (t_total > 0 && !ctx->o_orient.empty()) {
    TmxMatSet avg = {};
    avg.src[0] = (const cplx *)ctx->T.p;
    avg.dst[0] = (cplx *)ctx->Ta.p;
    // (the entries between the parity classes stay zero)
    CK(cudaMemsetAsync(ctx->Ta.p, 0, t_total * sizeof(cplx), st));
    if ((rc = launch_orient(ctx, avg, 1, ncoef, 0))) {
      return rc;
    }
    std::swap(ctx->T, ctx->Ta);
  }
  CK(cudaStreamSynchronize(st));
  ctx->t_averaged = true;
  ++ctx->batch_seq;
  ctx->sink_done = 0; // the T-matrices a sink holds are the unaveraged ones
  return TMX_OK;
}

extern "C" int tmx_batch_scattering_matrix(
    tmx_ctx *ctx, int64_t njobs, const int64_t *grain, const double *alpha,
    const double *beta, const double *theta_in, const double *phi_in,
    const double *theta_out, const double *phi_out, double *Z, double *S) {
  if (!ctx || njobs < 0 || (njobs > 0 && (!grain || !alpha || !beta || !theta_in ||
                                          !phi_in || !theta_out || !phi_out ||
                                          (!Z && !S)))) {
    return TMX_ERR_INVALID;
  }
  int rc;
  if ((rc = check_jobs(ctx, njobs, grain))) {
    return rc;
  }
  CK(cudaSetDevice(ctx->device));
  std::vector<zc> SL;
  if ((rc = lab_amplitudes(ctx, njobs, grain, alpha, beta, theta_in, phi_in,
                           theta_out, phi_out, SL))) {
    return rc;
  }
  for (int64_t j = 0; j < njobs; ++j) {
    const zc M[2][2] = {{SL[4 * j], SL[4 * j + 1]}, {SL[4 * j + 2], SL[4 * j + 3]}};
    if (Z) {
      z_from_s(M, Z + 16 * j);
    }
    if (S) {
      for (int q = 0; q < 4; ++q) {
        S[8 * j + 2 * q] = SL[4 * j + q].real();
        S[8 * j + 2 * q + 1] = SL[4 * j + q].imag();
      }
    }
  }
  return TMX_OK;
}

extern "C" int tmx_batch_extinction_matrix(tmx_ctx *ctx, int64_t njobs,
                                           const int64_t *grain,
                                           const double *alpha,
                                           const double *beta,
                                           const double *theta,
                                           const double *phi, double *K) {
  if (!ctx || njobs < 0 ||
      (njobs > 0 && (!grain || !alpha || !beta || !theta || !phi || !K))) {
    return TMX_ERR_INVALID;
  }
  int rc;
  if ((rc = check_jobs(ctx, njobs, grain))) {
    return rc;
  }
  CK(cudaSetDevice(ctx->device));
  std::vector<zc> SL;
  if ((rc = lab_amplitudes(ctx, njobs, grain, alpha, beta, theta, phi, theta,
                           phi, SL))) {
    return rc;
  }
  for (int64_t j = 0; j < njobs; ++j) {
    const zc M[2][2] = {{SL[4 * j], SL[4 * j + 1]}, {SL[4 * j + 2], SL[4 * j + 3]}};
    k_from_s(ctx->up_grains[grain[j]].k, M, K + 16 * j);
  }
  return TMX_OK;
}

extern "C" int tmx_batch_absorption_cross_sections(tmx_ctx *ctx, int64_t grain,
                                                   int32_t ntheta,
                                                   const double *theta,
                                                   int32_t ngauss, double *out) {
  if (!ctx || ntheta < 0 || ngauss < 1 || (ntheta > 0 && (!theta || !out))) {
    return TMX_ERR_INVALID;
  }
  int rc;
  if ((rc = check_jobs(ctx, 1, &grain))) {
    return rc;
  }
  CK(cudaSetDevice(ctx->device));
  return absorption(ctx, (int32_t)grain, ntheta, theta, ngauss, out);
}

extern "C" int tmx_batch_average_absorption_cross_section(tmx_ctx *ctx,
                                                          int64_t grain,
                                                          int32_t ngauss,
                                                          double *out) {
  if (!ctx || ngauss < 1 || !out) {
    return TMX_ERR_INVALID;
  }
  int rc;
  if ((rc = check_jobs(ctx, 1, &grain))) {
    return rc;
  }
  CK(cudaSetDevice(ctx->device));
  // TMatrix::get_average_absorption_cross_section (TMatrix.hpp:2260-2287)
  std::vector<double> ct(ngauss), wt(ngauss), tg(ngauss), cabs(2 * ngauss);
  tmx_host_gauss_legendre(ngauss, ct.data(), wt.data());
  for (int i = 0; i < ngauss; ++i) {
    tg[i] = acos(ct[i]);
  }
  if ((rc = absorption(ctx, (int32_t)grain, ngauss, tg.data(), ngauss, cabs.data()))) {
    return rc;
  }
  double result = 0.;
  for (int i = 0; i < ngauss; ++i) {
    result += cabs[2 * i] * wt[i];
  }
  *out = 0.5 * result;
  return TMX_OK;
}
