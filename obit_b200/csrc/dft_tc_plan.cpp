// Host planning of the tensor-core form (dft_tc.cu): uniformly spaced runs of
// the selected channels, the warps' grids of rows x columns, the exponent
// tables and their bounds, and the choice between this form and the
// recurrence kernels.  Plain C++, no CUDA calls.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <map>

#include "dft_tc.h"

namespace obit {

namespace {

// Largest neglected relative amplitude of a term (the corner of a segment's
// grid; a fifth of it or less in the mean square): the rank-one residual
// (alpha - alpha_t) R without the cross product, and the second order of the
// cross exponent with it.
constexpr double kTcResidualTol = 2.5e-6;
// Without the cross product the exponents (alpha - alpha_t) lam of rows and
// columns are taken to first order: x^2 / 2 at most this.
constexpr double kTcFirstTol = 1.5e-7;

struct Run {
  double f0, df;  // frequency ratios f0 + k df
  int list0, n;   // channel-list range
  double lnShift; // log-frequency term = ln f + lnShift
  int jplane;
};

void split_ds(double x, float* hi, float* lo) {
  *hi = (float)x;
  *lo = (float)(x - (double)*hi);
}

// Cost of one team per 8 components in scheduler cycles of the chip, from the
// measured rates of full teams of points (1024, 512, 256 and 128 channels: 11.3,
// 10.8, 8.6 and 5.8 T evaluations/s), against kRecurCost per channel of
// the recurrence kernels' blocks (4.6-4.8 T).  With a spectral index the shapes measured 7.5,
// 7.3, 6.8 and 4.7 T, in the same order.
struct Shape {
  int MA, NJ, T;
  double cost;
};
// A beam's column groups are its correlations (4 or 2).
constexpr Shape kBeamShapes4[] = {{2, 4, 1, 700.0}, {1, 4, 1, 420.0}};
constexpr Shape kBeamShapes2[] = {{2, 2, 1, 420.0}};
constexpr Shape kShapes[] = {{2, 2, 2, 792.0}, {2, 2, 1, 416.0}, {1, 2, 1, 261.0}, {1, 1, 1, 192.0}};
constexpr double kRecurCost = 1.9, kRecurShort = 3.25;

bool tab_kind(int kind) { return kind == kPointTSpec || kind == kGaussTSpec; }
bool spec_kind(int kind) { return kind == kPointSpec || kind == kGaussSpec || tab_kind(kind); }
bool gauss_kind(int kind) { return kind == kGauss || kind == kGaussSpec || kind == kGaussTSpec; }

// Half the largest spread of the spectral index within a chunk.
double chunk_spread(const float* table, int stride, int field, int ncomp) {
  double s = 0.0;
  for (int c0 = 0; c0 < ncomp; c0 += kTcChunk) {
    const int c1 = std::min(ncomp, c0 + kTcChunk) - 1;
    const double at = 0.5 * ((double)table[(size_t)c0 * stride + field] + (double)table[(size_t)c1 * stride + field]);
    for (int c = c0; c <= c1; c++) s = std::max(s, std::fabs((double)table[(size_t)c * stride + field] - at));
  }
  return s;
}

double max_abs(const float* table, int stride, int field, int ncomp) {
  double s = 0.0;
  for (int c = 0; c < ncomp; c++) s = std::max(s, std::fabs((double)table[(size_t)c * stride + field]));
  return s;
}

}  // namespace

double tc_recur_cost(const Plan& recur) {
  // rows of one or two blocks leave its prologues little to share: 2.7 T on
  // 64-channel rows of points, against 2.8 T here
  if (recur.model.kind == kPoint && recur.kp.nblocks <= 2 && recur.tune.K == 32) {
    int n = 0;
    for (const BlockDesc& b : recur.blocks) n += b.len;
    return kRecurShort * n;
  }
  return kRecurCost * recur.kp.nblocks * recur.tune.K;  // its blocks are padded too
}

void tc_plan_layout(const LayoutDesc& L, const ModelDesc& M, const std::function<const float*()>& fetch,
                    double recurCost, std::vector<TcPlan>* plan, const int* jchan, int ncorr) {
  plan->clear();
  const bool beam = jchan != nullptr;
  const bool spec = spec_kind(M.kind), gauss = gauss_kind(M.kind), tab = tab_kind(M.kind);
  if (!(M.kind == kPoint || M.kind == kGauss || tab || (spec && M.nterm == 1)) || (tab && beam)) return;
  const int npt = M.ncompPt, ntot = npt + M.ncomp;
  if (ntot < kTcMinComps || M.ncomp < 1) return;
  const int stride = comp_stride(M);
  const int planes = tab ? M.nspec : 0;
  const int used = (gauss ? (spec ? 8 : 7) : (spec ? 5 : 4)) + planes;
  // ---- uniformly spaced runs of the selected channels -------------------------
  std::vector<Run> runs;
  std::vector<double> f;
  std::vector<int> off;
  std::vector<double> ln;
  std::vector<int> jp, pl;
  for (int iIF = L.ifb; iIF <= L.ife; iIF++)
    for (int ch = L.chanb; ch <= L.chane; ch++) {
      const int i = ch * L.kincf + iIF * L.kincif;
      f.push_back(L.fscale[i]);
      off.push_back(L.nrparm + iIF * L.incif + ch * L.incf + (beam ? 0 : L.stokb * L.incs));
      jp.push_back(beam ? jchan[i] : 0);
      pl.push_back(tab ? L.specIndex[i] : 0);
      if (tab && (pl.back() < 0 || pl.back() >= planes)) return;
      ln.push_back(spec ? L.lnspec[i] : 0.0);
      if (!(L.fscale[i] > 0.0)) return;
    }
  const int n = (int)f.size();
  for (int i = 0; i < n;) {
    int e = i + 1;
    double df = 0.0;
    if (e < n && jp[e] == jp[i]) {
      df = f[e] - f[i];
      // the increment's own rounding grows with the run; the run is checked
      // against its mean increment below
      while (e < n && jp[e] == jp[i] && std::fabs(f[e] - (f[i] + (e - i) * df)) <= (1e-13 + 4.5e-16 * (e - i)) * f[i]) e++;
    }
    // a row of D = 8 or 16 channels lies in one coarse plane: a run ends where
    // the plane changes inside one
    for (int k = i + 1; k < e; k++)
      if (pl[k] != pl[k - 1] && (k - i) % 16 != 0) e = k;
    Run r{f[i], df, i, e - i, spec ? ln[i] - std::log(f[i]) : 0.0, jp[i]};
    if (r.n > 1) r.df = (f[e - 1] - f[i]) / (r.n - 1);
    for (int k = 0; k < r.n; k++) {
      if (std::fabs(f[i + k] - (r.f0 + k * r.df)) > 2e-13 * f[i]) return;
      if (spec && !tab && std::fabs(ln[i + k] - (std::log(f[i + k]) + r.lnShift)) > 1e-9) return;
    }
    runs.push_back(r);
    i = e;
  }

  // ---- the cheapest cover of every run by the shapes ------------------------------
  std::vector<Shape> fit;
  if (!beam)
    for (const Shape& s : kShapes) fit.push_back(s);
  else if (ncorr > 2)
    for (const Shape& s : kBeamShapes4) fit.push_back(s);
  else
    for (const Shape& s : kBeamShapes2) fit.push_back(s);
  auto capacity = [&](const Shape& s) { return 128 * s.MA * (beam ? 1 : s.NJ) * s.T; };
  struct Piece {
    int run, t0;
  };
  std::vector<std::vector<Piece>> use;
  auto cover_runs = [&]() -> double {  // fills use (pieces per shape), returns the cost
    std::map<int, std::pair<double, int>> cover;  // channels left -> (cost, shape)
    cover[0] = {0.0, -1};
    std::function<double(int)> cheapest = [&](int left) -> double {
      auto it = cover.find(left);
      if (it != cover.end()) return it->second.first;
      std::pair<double, int> best{1e300, -1};
      for (size_t i = 0; i < fit.size(); i++) {
        const double c = fit[i].cost + cheapest(std::max(0, left - capacity(fit[i])));
        if (c < best.first) best = {c, (int)i};
      }
      cover[left] = best;
      return best.first;
    };
    double cost = 0.0;
    use.assign(fit.size(), {});
    for (size_t i = 0; i < runs.size(); i++) {
      cost += cheapest(runs[i].n);
      for (int t0 = 0; t0 < runs[i].n;) {
        const int k = cover[runs[i].n - t0].second;
        use[k].push_back({(int)i, t0});
        t0 += capacity(fit[k]);
      }
    }
    return cost;
  };
  for (const Run& r : runs)
    if (r.n > 65536) return;
  if (!(cover_runs() < recurCost)) return;  // before the table is looked at

  const float* table = fetch();
  if (!table) return;
  for (int c = 0; c < ntot; c++) {
    const float* r = table + (size_t)c * stride;
    const int nf = c < npt ? 5 + planes : used;
    for (int i = 0; i < nf; i++)
      if (!std::isfinite(r[i])) return;
    // a taper never grows: g1 u^2 + g2 v^2 + g3 u v <= 0 for every u, v
    if (gauss && c >= npt && !(r[4] <= 0.f && r[5] <= 0.f && 4.0 * r[4] * r[5] >= (double)r[6] * r[6] * (1.0 - 1e-5)))
      return;
  }

  // ---- bounds and tables ------------------------------------------------------------
  const double spreadPt = (gauss && npt) || (!gauss && spec)
                              ? chunk_spread(table, stride, kSpecIndexField, gauss ? npt : M.ncomp) : 0.0;
  const float* gt = table + (size_t)npt * stride;
  const double spreadG = (gauss && spec) ? chunk_spread(gt, stride, 7, M.ncomp) : 0.0;
  double amax = 0.0;
  if (!gauss && spec) amax = max_abs(table, stride, kSpecIndexField, M.ncomp);
  if (gauss && npt) amax = max_abs(table, stride, kSpecIndexField, npt);
  if (gauss && spec) amax = std::max(amax, max_abs(gt, stride, 7, M.ncomp));
  // Teams of shape s over pieces of runs; false when a bound fails.
  auto build = [&](const Shape& s, const std::vector<Piece>& pieces, TcPlan* out) -> bool {
    const int NC = beam ? 1 : s.NJ, segCap = 128 * s.MA * NC;
    TcPlan p;
    p.MA = s.MA;
    p.NJ = s.NJ;
    p.T = s.T;
    p.NC = NC;
    p.beam = beam;
    p.kind = M.kind;
    p.mixed = npt > 0;
    p.chanOff = off;
    const TcExpo lay = tc_expo_layout(s.MA, NC);
    const int D = 8 * NC, a0 = 8 * (s.MA - 1) + 4, rows = 16 * s.MA, cols = 8 * NC;
    const double inv2pi = 0.15915494309189533577;
    double resid1 = 0.0, resid2 = 0.0, gcross = 0.0, range = 0.0;
    for (const Piece& pc : pieces) {
      const Run& r = runs[pc.run];
      const int t0 = pc.t0;
      {
        TcTeamDesc tm{};
        tm.D = D;
        split_ds(D * r.df * inv2pi, &tm.w_hi, &tm.w_lo);
        split_ds(8.0 * D * r.df * inv2pi, &tm.w8_hi, &tm.w8_lo);
        split_ds(r.df * inv2pi, &tm.s_hi, &tm.s_lo);
        for (int q = 0; q < s.T; q++) {
          TcSeg& g = tm.seg[q];
          const int k0 = t0 + q * segCap;
          auto F = [&](double x) { return r.f0 + (k0 + x) * r.df; };  // ratio at channel offset x of the segment
          g.end = r.list0 + std::min(r.n, k0 + segCap);
          split_ds(F(D * a0 + 4) * inv2pi, &g.fa_hi, &g.fa_lo);
          g.ch0 = r.list0 + k0;
          g.jplane = r.jplane;
          if (!(spec || gauss) || k0 >= r.n) continue;
          if (!(std::min(F(0), F(segCap - 1)) > 0.05 * r.f0)) return false;
          // exponent tables: rows a against the middle column, columns n against the middle row
          g.expo = (int)p.expo.size();
          p.expo.resize(p.expo.size() + lay.total, 0.0f);
          float* ex = p.expo.data() + g.expo;
          const double nm = 0.5 * (cols - 1);
          // log-frequency term, the row's coarse plane taken from its first channel
          const int last = std::min(r.n - k0, segCap) - 1;          // last valid channel offset
          auto at = [&](double a) { return r.list0 + k0 + std::min<int>(D * (int)a, last); };
          auto smooth = [&](double a, double nn) { return std::log(F(D * a + nn)); };
          auto Lg = [&](double a, double nn) {
            return smooth(a, nn) + (tab ? ln[at(a)] - std::log(f[at(a)]) : r.lnShift);
          };
          auto F2 = [&](double a, double nn) { const double x = F(D * a + nn); return x * x; };
          const double ar = r.df >= 0.0 ? 0.0 : (double)(last / D);  // row of the least taper
          const double am = 0.5 * std::min<double>(rows - 1, (double)(last / D));  // middle valid row
          const double lam0 = tab ? 0.0 : Lg(am, nm), xi0 = F2(ar, nm);
          g.lam0 = (float)lam0;
          g.xi0 = (float)xi0;
          double yy = 0.0;
          for (int c = 0; c < cols; c++) {
            const double y = (c - nm) * r.df;
            ex[lay.y + c] = (float)y;
            ex[lay.lamCol + c] = spec ? (float)(smooth(am, c) - smooth(am, nm)) : 0.f;
            ex[lay.xiCol + c] = (float)(F2(am, c) - F2(am, nm));
            yy += y * y;
          }
          g.plane0 = g.plane1 = pl[at(0)];
          for (int a = 0; a < rows; a++) {
            const int plane = pl[at(a)];
            g.plane0 = std::min(g.plane0, plane);
            g.plane1 = std::max(g.plane1, plane);
            std::memcpy(&ex[lay.plane + a], &plane, sizeof(int));
            ex[lay.lamRow + a] = spec ? (float)(Lg(a, nm) - lam0) : 0.f;
            ex[lay.xiRow + a] = (float)(F2(a, nm) - xi0);
            ex[lay.xf + a] = (float)(2.0 * D * (a - am) * r.df);
            double ry = 0.0, R[64];
            for (int c = 0; c < cols && spec; c++) {
              R[c] = smooth(a, c) - smooth(a, nm) - smooth(am, c) + smooth(am, nm);
              ry += R[c] * (c - nm) * r.df;
              // fragment order: lane (row % 8) * 4 + (column % 8) / 2
              const int mi = a >> 4, e = 2 * ((a >> 3) & 1) + (c & 1);
              const int lane = 4 * (a & 7) + ((c & 7) >> 1);
              ex[lay.L + ((mi * NC + (c >> 3)) * 32 + lane) * 4 + e] = (float)(Lg(a, c) - lam0);
            }
            const double xl = (spec && yy > 0.0) ? ry / yy : 0.0;
            ex[lay.xl + a] = (float)xl;
            for (int c = 0; c < cols; c++) {
              if (D * a + c > last) continue;
              const double y = (c - nm) * r.df;
              if (spec) {
                resid1 = std::max(resid1, std::fabs(R[c]));
                resid2 = std::max(resid2, std::fabs(R[c] - xl * y));
                range = std::max(range, std::fabs(Lg(a, c) - lam0));
              }
              gcross = std::max(gcross, std::fabs(2.0 * D * (a - am) * r.df * y) / F2(a, c));
            }
          }
        }
        p.teams.push_back(tm);
      }
    }
    auto second = [&](double x) { return 0.5 * x * x; };
    if (spec && amax * range > 8.0) return false;
    if ((!gauss && spec) || npt) {
      p.crossPt = spreadPt * resid1 > kTcResidualTol || second(spreadPt * range) > kTcFirstTol;
      if (p.crossPt && std::max(spreadPt * resid2, second(spreadPt * resid1)) > kTcResidualTol) return false;
    }
    if (gauss) {
      // second order of the taper's cross exponent q c times the taper exp(-q): largest at q = 2
      if (0.2707 * gcross * gcross > kTcResidualTol) return false;
      if (spec && std::max(spreadG * resid2, second(spreadG * resid1)) > kTcResidualTol) return false;
    }
    p.on = true;
    *out = std::move(p);
    return true;
  };

  // a shape that fails a bound is left out and the runs covered by the others
  while (!fit.empty() && cover_runs() < recurCost) {
    std::vector<TcPlan> parts;
    size_t bad = fit.size();
    for (size_t k = 0; k < fit.size() && bad == fit.size(); k++) {
      if (use[k].empty()) continue;
      TcPlan p;
      if (build(fit[k], use[k], &p)) parts.push_back(std::move(p));
      else bad = k;
    }
    if (bad == fit.size()) {
      *plan = std::move(parts);
      return;
    }
    fit.erase(fit.begin() + bad);
  }
}

}  // namespace obit
