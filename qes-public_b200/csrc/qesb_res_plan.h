// Plans of the resident solves (qesb_sor_res.cu), as host arithmetic alone: how
// a domain is cut into tiles, which launches a list of domains takes, and which
// of a batch's domains are solved that way.
#pragma once
#include <algorithm>
#include <functional>
#include <map>
#include <queue>
#include <tuple>
#include <utility>
#include <vector>

namespace qesb {

constexpr int kResThreads = 512;       // one CTA per SM
constexpr int kResSmemBytes = 230400;  // the per-block limit less the kernel's static part
constexpr int kResMaxLaunches = 16;    // launches of one batch (group sizes)

struct ResSize {
  int X, Y, Z;  // cells
};

// Tiles of a resident solve over at most so many CTAs, with the estimated
// cycles of a half-sweep; nty = 0: the domain does not fit.
struct ResPlan {
  int nty = 0, ntz = 0;
  int tym = 0, tzm = 0;  // the largest tile
  double cost = 0;
};

// The estimate: row steps of the CTA's warps (350 cycles for all of them, dearer
// where R streams from L2) and the exchange. Measured solves take 1.45 (the
// smallest domains) to 1.95 times it: 1.85, at 1.9 GHz, in kResUs.
constexpr double kResUs = 2 * 1.85 / 1900.0;  // microseconds an iteration per estimated cycle of a half-sweep
inline ResPlan res_plan(const ResSize &G, int ctas)
{
  constexpr int NW = kResThreads / 32;
  ResPlan best;
  const int nq4 = ((G.X + 1) / 2 + 3) / 4, P = 4 * nq4, rows = G.Y - 2, planes = G.Z - 2;
  const long cap = kResSmemBytes / 4;
  // for each cut along z the most tiles along y that the CTAs allow (no more than their row count needs)
  for (int ntz = 1; ntz <= std::min(planes, ctas); ++ntz) {
    const int tz = (planes + ntz - 1) / ntz, ty = (rows + std::min(rows, ctas / ntz) - 1) / std::min(rows, ctas / ntz);
    const int nty = (rows + ty - 1) / ty;
    const long base = 2048 + 72L * tz + 2L * (tz + 2) * (ty + 2) * P + 2L * tz * ty * nq4 + 4L * (tz + ty) * nq4 + 8;
    if (base > cap) continue;
    const int rp = (int)std::min<long>(tz, (cap - base) / (2L * ty * P));
    const int ch = ((tz + 1) / 2 * nq4 + 31) / 32 + (tz / 2 * nq4 + 31) / 32;  // warps' columns
    int steps = 1 << 30;
    for (int n = 1; n <= std::min(ty, 32); ++n) steps = std::min(steps, (ch * n + NW - 1) / NW * ((ty + n - 1) / n + 4));
    const double step = 350.0 * (1.0 + 0.4 * (tz - rp) / tz);
    const double comm = nty * ntz > 1 ? 2000.0 + 0.25 * (tz + ty) * nq4 : 200.0;
    const double cost = step * steps + comm;
    if (best.nty == 0 || cost < best.cost) {
      best.nty = nty;
      best.ntz = ntz;
      best.cost = cost;
      best.tym = ty;
      best.tzm = tz;
    }
  }
  return best;
}

// Plans by grid and CTAs, each made once. Bounded: a launch of many more grids
// than this makes them again.
struct ResPlans {
  std::map<std::tuple<int, int, int>, std::vector<std::pair<int, ResPlan>>> of_grid;
  ResPlan of(const ResSize &G, int ctas)
  {
    if (of_grid.size() > 2048) of_grid.clear();
    auto &v = of_grid[{G.X, G.Y, G.Z}];
    for (const auto &p : v)
      if (p.first == ctas) return p.second;
    v.emplace_back(ctas, res_plan(G, ctas));
    return v.back().second;
  }
};

// The launches of a list of domains: domains of about the same best group size
// go together, large ones first.
struct ResLaunch {
  int first, n, groups, gsz;  // of `order`
};
struct ResSchedule {
  std::vector<int> order;
  std::vector<ResLaunch> launches;
  double cost = 0;           // estimated cycles of a half-sweep of all domains
  std::vector<double> each;  // a domain's own share of it
};

// The SMs are split into g groups of sms / g CTAs. Of the counts with the same
// group size the largest is never worse, so only those are looked at (23 of
// 148): with every count, and plans looked up for each, the schedule of 256
// uneven small domains took 100 ms of host time a batch, now 2.
inline ResSchedule res_schedule(ResPlans &plans, const std::vector<ResSize> &ds, int sms)
{
  const int n = (int)ds.size();
  ResSchedule r;
  r.order.resize(n);
  r.each.resize(n);
  std::vector<int> sizes, most;  // group sizes, largest first, and the most groups of each
  for (int g = 1; g <= std::min(n, sms); ++g) {
    if (sizes.empty() || sizes.back() != sms / g) {
      sizes.push_back(sms / g);
      most.push_back(g);
    }
    most.back() = g;
  }
  const int nc = (int)sizes.size();
  std::vector<double> cost((size_t)n * nc, -1.0);  // -1: does not fit
  std::vector<int> ng(n);
  for (int i = 0; i < n; ++i) {
    r.order[i] = i;
    for (int c = 0; c < nc; ++c) {
      const ResPlan p = plans.of(ds[i], sizes[c]);
      if (!p.nty) break;
      cost[(size_t)i * nc + c] = p.cost;
      if (ng[i] == 0 || p.cost / most[c] < r.each[i]) {
        r.each[i] = p.cost / most[c];
        ng[i] = most[c];
      }
    }
  }
  std::stable_sort(r.order.begin(), r.order.end(), [&](int a, int b) {
    if (ng[a] != ng[b]) return ng[a] < ng[b];
    return (long)ds[a].X * ds[a].Y * ds[a].Z > (long)ds[b].X * ds[b].Y * ds[b].Z;
  });
  // the time of one launch of order[i, j) in g groups of sizes[c]: each takes the next domain when it is free
  auto span = [&](int i, int j, int c, int g, double limit) {
    std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
    double last = 0.0, sum = 0.0;
    for (int q = i; q < j; ++q) {
      const double d = cost[(size_t)r.order[q] * nc + c];
      if (d < 0) return -1.0;
      sum += d;
      if (limit > 0 && sum / g >= limit) return limit;  // not shorter
      double t = d;
      if ((int)free_at.size() == g) {
        t += free_at.top();
        free_at.pop();
      }
      free_at.push(t);
      last = std::max(last, t);
    }
    return last;
  };
  auto best_launch = [&](int i, int j, double *cost_) {
    ResLaunch l{i, j - i, 1, sms};
    *cost_ = span(i, j, 0, 1, 0.0);
    for (int c = 0; c < nc; ++c) {
      const int g = std::min(most[c], j - i);
      if (g < 2) continue;
      if (sms / g != sizes[c]) break;  // more groups than domains
      const double t = span(i, j, c, g, *cost_);
      if (t < 0) break;
      if (t < *cost_) {
        *cost_ = t;
        l.groups = g;
        l.gsz = sizes[c];
      }
    }
    return l;
  };
  double before = 0;  // the last launch's
  for (int i = 0; i < n;) {
    int j = i;
    while (j < n && ng[r.order[j]] == ng[r.order[i]]) ++j;
    double c = 0;
    const ResLaunch l = best_launch(i, j, &c);
    if (!r.launches.empty()) {  // together with the launch before where that is shorter (or there are many)
      double cm = 0;
      const ResLaunch m = best_launch(r.launches.back().first, j, &cm);
      if (cm <= before + c || (int)r.launches.size() == kResMaxLaunches) {
        r.launches.back() = m;
        r.cost += cm - before;
        before = cm;
        i = j;
        continue;
      }
    }
    r.launches.push_back(l);
    r.cost += c;
    before = c;
    i = j;
  }
  return r;
}

// Microseconds that a domain adds to an iteration of the streaming list sweeps
// (measured: 3.0 a million cells on full 128-cell row tiles, 4.5 where half of a
// tile is empty), and what the list's launches take of themselves.
inline double list_us(const ResSize &G)
{
  const int qn = (G.X + 1) / 2;
  return 3.0e-6 * (double)((long)G.X * G.Y) * G.Z * 0.5 * (1.0 + 128.0 * ((qn + 127) / 128) / qn);
}
constexpr double kListUs = 12.0;

// Which domains of a batch take the resident kernel, of those that may: all,
// none, or those it is faster for than their part of the list sweeps, by the
// shorter estimate. A list of small domains gains the most (16 of 64 x 64 x 32:
// 10 against 35 us an iteration; 16 of 128 x 128 x 48: 42 against 76), many
// large ones (16 of 192 x 192 x 64: 171 against 133) stay with the list sweeps.
struct ResChoice {
  std::vector<char> is_res;  // by domain
  ResSchedule sched;         // of those, in turn
};
inline ResChoice res_choose(ResPlans &plans, const std::vector<ResSize> &ds, const std::vector<char> &may, int sms)
{
  const int n = (int)ds.size();
  std::vector<ResSize> all;
  std::vector<int> of;
  double others = 0;  // list time of the domains that have no choice
  for (int i = 0; i < n; ++i) {
    if (may[i]) {
      all.push_back(ds[i]);
      of.push_back(i);
    } else {
      others += list_us(ds[i]);
    }
  }
  ResChoice r;
  r.is_res.assign(n, 0);
  if (all.empty()) return r;
  ResSchedule sch = res_schedule(plans, all, sms), part_sch;
  double list_all = 0, list_rest = 0;
  std::vector<char> some(n, 0);
  std::vector<ResSize> part;
  for (size_t q = 0; q < all.size(); ++q) {
    const double l = list_us(all[q]);
    list_all += l;
    if (kResUs * sch.each[q] < l) {
      some[of[q]] = 1;
      part.push_back(all[q]);
    } else {
      list_rest += l;
    }
  }
  const auto list = [&](double us) { return us + others > 0 ? us + others + kListUs : 0.0; };
  const double t_all = kResUs * sch.cost + list(0.0), t_none = list(list_all);
  double t_some = t_none;
  if (part.size() == all.size()) {
    t_some = t_all;
  } else if (!part.empty()) {
    part_sch = res_schedule(plans, part, sms);
    t_some = kResUs * part_sch.cost + list(list_rest);
  }
  if (t_none <= t_all && t_none <= t_some) return r;
  if (t_all <= t_some) {
    r.is_res = may;
    r.sched = std::move(sch);
  } else {
    r.is_res = some;
    r.sched = std::move(part_sch);
  }
  return r;
}

}  // namespace qesb
