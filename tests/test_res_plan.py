"""The host's plans of resident solves (csrc/qesb_res_plan.h): the launches of a
list of domains against a search over every group count, the plans' limits, and
the host time that a batch of many different domains spends on them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "qesb_res_plan.h"
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>
using namespace qesb;
constexpr int SMS = 148;

// the shortest launch of the domains `o` by greedy dispatch, over every number of groups
double brute(const std::vector<ResSize> &ds, const std::vector<int> &o)
{
  double best = -1;
  for (int g = 1; g <= std::min((int)o.size(), SMS); ++g) {
    std::vector<double> t(g, 0.0);
    for (int q : o) {
      const ResPlan p = res_plan(ds[q], SMS / g);
      if (!p.nty) return best;
      *std::min_element(t.begin(), t.end()) += p.cost;
    }
    const double c = *std::max_element(t.begin(), t.end());
    if (best < 0 || c < best) best = c;
  }
  return best;
}

int main()
{
  std::mt19937 r(1);
  int bad = 0, resident = 0;
  for (int n : {1, 2, 3, 7, 12, 30, 60}) for (int rep = 0; rep < 12; ++rep) {
    std::vector<ResSize> ds;
    const int top = 20 + 60 * (rep % 4);
    for (int i = 0; i < n; ++i) ds.push_back({3 + (int)(r() % top), 3 + (int)(r() % top), 3 + (int)(r() % 40)});
    std::vector<char> may(n);
    for (int i = 0; i < n; ++i) may[i] = res_plan(ds[i], SMS).nty > 0 && r() % 8 != 0;
    ResPlans plans;
    const ResChoice c = res_choose(plans, ds, may, SMS);
    std::vector<ResSize> in;
    for (int i = 0; i < n; ++i) {
      bad += c.is_res[i] && !may[i];
      if (c.is_res[i]) in.push_back(ds[i]);
    }
    resident += in.size();
    std::vector<int> seen(in.size(), 0);
    double cost = 0;
    bad += (int)c.sched.launches.size() > kResMaxLaunches;
    for (const ResLaunch &l : c.sched.launches) {
      bad += l.groups < 1 || l.gsz < 1 || l.groups * l.gsz > SMS;
      std::vector<int> o(c.sched.order.begin() + l.first, c.sched.order.begin() + l.first + l.n);
      for (int q : o) {
        ++seen[q];
        const ResPlan p = plans.of(in[q], l.gsz);
        const int rows = in[q].Y - 2, planes = in[q].Z - 2;
        bad += p.nty < 1 || p.nty * p.ntz > l.gsz || p.nty > rows || p.ntz > planes;
        bad += p.tym * p.nty < rows || p.tzm * p.ntz < planes;
      }
      cost += brute(in, o);
    }
    for (int s : seen) bad += s != 1;
    bad += std::fabs(cost - c.sched.cost) > 1e-9 * cost;
  }
  // many uneven small domains, each batch call anew
  std::vector<ResSize> ds;
  for (int i = 0; i < 256; ++i) ds.push_back({48 + (int)(r() % 48), 48 + (int)(r() % 48), 24 + (int)(r() % 16)});
  ResPlans plans;
  double ms = 1e30;
  for (int rep = 0; rep < 5; ++rep) {
    const auto t0 = std::chrono::steady_clock::now();
    res_choose(plans, ds, std::vector<char>(256, 1), SMS);
    ms = std::min(ms, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
  }
  std::printf("%d %d %.3f\n", bad, resident, ms);
}
"""


@pytest.fixture(scope="module")
def result(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "plan.cpp", d / "plan"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "qes-public_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    bad, resident, ms = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    return int(bad), int(resident), float(ms)


def test_schedules_are_whole_and_the_shortest_by_group_count(result):
    assert result[0] == 0 and result[1] > 0


def test_a_large_batch_costs_little_host_time(result):
    """Some 2 ms; looking at every group count and looking each plan up took 100."""
    assert result[2] < 30.0
