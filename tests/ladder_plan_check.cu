// Host check of the ladder kernels' task lists (built by tests/test_ladder_plan.py; runs without a GPU): every
// index that ladder_path_kernel, ladder_close_kernel, ladder_gather_kernel and ladder_back_kernel read from a
// plan lies inside its array, and what a task loads was stored before.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <memory>
#include <numeric>
#include <string>
#include <vector>

#include "../graph-vqe_b200/csrc/common.cuh"
#include "../graph-vqe_b200/csrc/evolve.cuh"
#include "../graph-vqe_b200/csrc/expect.cuh"
#include "../graph-vqe_b200/csrc/gradient.cuh"
#include "../graph-vqe_b200/csrc/ladder.cuh"
#include "../graph-vqe_b200/csrc/ladder_grad.cuh"
using namespace vqemps;
#include "../graph-vqe_b200/csrc/ladder_plan.inc"
#include "../graph-vqe_b200/csrc/ladder_grad_plan.inc"

static std::string fault;
static bool need(bool ok, const char *what, long long at) {
  if (!ok && fault.empty()) fault = std::string(what) + " at " + std::to_string(at);
  return ok;
}

// One launch as ladder_path_kernel walks it; stored: slots of earlier launches per half, updated.
static void walk(const std::vector<LadTask> &tasks, const std::vector<uint32_t> &steps, const std::vector<int32_t> &slots,
                 const LadderLaunch &ln, const int (&nslot)[2], std::vector<uint8_t> (&stored)[2], int n) {
  std::vector<uint8_t> now[2] = {std::vector<uint8_t>(nslot[0], 0), std::vector<uint8_t>(nslot[1], 0)};
  for (int i = 0; i < ln.ntasks; ++i) {
    const LadTask &t = tasks[ln.first + i];
    const int half = i < ln.npre ? 0 : 1;
    need(((t.flags >> 1) & 1) == half, "half of task", i);
    need(t.step >= 0 && t.nsteps >= 0 && (size_t)t.step + t.nsteps <= steps.size(), "steps of task", i);
    std::vector<uint8_t> mine(nslot[half], 0);
    size_t at = t.slot;
    auto read = [&] {                                // the kernel reads the next entry ahead of its use
      if (need(at < slots.size(), "slot entry", (long long)at)) return slots[at];
      return (int32_t)0;
    };
    int32_t slot = read();
    auto advance = [&] { ++at; slot = read(); };
    auto inside = [&] { return need(slot >= 0 && slot < nslot[half], "slot of task", i); };
    auto store = [&] {
      if (!inside()) return;
      need(!now[half][slot] || mine[slot], "slot stored by two tasks", slot);
      now[half][slot] = mine[slot] = 1;
      advance();
    };
    if (t.flags & 8) store();
    for (int s = t.step; s < t.step + t.nsteps && fault.empty(); ++s) {
      need((int)(steps[s] >> 16) < n, "site of step", s);
      if (steps[s] & 32) {
        if (inside()) need(mine[slot] || stored[half][slot], "load before its store", slot);
        advance();
      }
      if (steps[s] & 4) store();
    }
  }
  for (int h = 0; h < 2; ++h)
    for (int s = 0; s < nslot[h]; ++s) stored[h][s] |= now[h][s];
}

static void check_grad(const LadderPlan &pl, int list, int n) {
  LadderGradPlan g;
  build_ladder_grad_plan(g, pl.words, pl.leaf_coef, LAD_SUBTREE[list]);
  const int nslot[2] = {g.nslot_p, g.nslot_s};
  std::vector<uint8_t> stored[2] = {std::vector<uint8_t>(nslot[0], 0), std::vector<uint8_t>(nslot[1], 0)};
  walk(g.tasks, g.steps, g.slots, g.launch, nslot, stored, n);
  for (const LadPair &p : g.pairs) {
    need(p.pslot >= 0 && p.pslot < nslot[0] && stored[0][p.pslot], "prefix of pair", p.pslot);
    need(p.sslot >= 0 && p.sslot < nslot[1] && stored[1][p.sslot], "suffix of pair", p.sslot);
    need(p.leaf >= 0 && p.leaf < pl.nleaf, "leaf of pair", p.leaf);
  }
  const int nc = (int)g.closers.size();
  auto closer = [&](const LadClose &c, int half, int sums) {       // half of the step: takes the other one's slots
    if (c.flags & 4) need(c.slot >= 0 && c.slot < sums, "sum of a closure", c.slot);
    else need(c.slot >= 0 && c.slot < nslot[1 - half] && stored[1 - half][c.slot], "slot of a closure", c.slot);
  };
  for (int i = 0; i < g.ngather; ++i) {
    const LadGather &s = g.gathers[i];
    if (need(s.first >= 0 && s.count > 0 && s.first + s.count <= nc, "words of sum", i))
      for (int c = 0; c < s.count; ++c) closer(g.closers[s.first + c], s.half, i < g.ngather1 ? 0 : g.ngather1);
  }
  need(g.back.size() == g.nsteps + 1 && g.steps.size() == g.nsteps, "step records", (long long)g.back.size());
  for (int i = 0; i < g.launch.ntasks && fault.empty(); ++i) {
    const LadTask &t = g.tasks[g.launch.first + i];
    const int half = i < g.launch.npre ? 0 : 1, ncot = half ? g.ncot_s : g.ncot_p;
    for (int s = t.step; s < t.step + t.nsteps; ++s) {
      const LadBack &b = g.back[s];
      need(b.in >= -1 && b.in < nslot[half], "input of step", s);
      need(b.cot_add >= -1 && b.cot_add < ncot, "cotangent of step", s);
      need(b.cot_out >= -2 && (b.cot_out >> 1) < ncot, "cotangent from step", s);
      if (need(b.close >= 0 && b.close <= g.back[s + 1].close && g.back[s + 1].close <= nc, "words of step", s))
        for (int c = b.close; c < g.back[s + 1].close; ++c) closer(g.closers[c], half, g.ngather);
    }
  }
  need((int)g.site_off.size() == 4 * n + 1 && g.site_off[4 * n] == (int)g.nsteps, "steps of sites", (long long)g.site_off.size());
  for (int32_t s : g.site_steps) need(s >= 0 && s < (int)g.nsteps, "step of a site", s);
}

// Returns the number of steps of the gradient's lists, or -1 with the first fault in msg[size].
extern "C" long long check_ladder_plan(int n, int T, const uint8_t *codes, const double *coeffs, int mirror, int real, int layers,
                                       char *msg, int size) {
  fault.clear();
  LadderCircuit lc;
  lc.mirror = mirror != 0;
  lc.real = real != 0;
  lc.layers = layers;
  LadderPlan pl;
  build_ladder_plan(pl, lc, n, T, std::vector<uint8_t>(codes, codes + (size_t)T * n), std::vector<double>(coeffs, coeffs + T));
  long long steps = 0;
  for (const LadderList &l : pl.lists) {
    const int nslot[2] = {pl.nslot_p, pl.nslot_s};
    std::vector<uint8_t> stored[2] = {std::vector<uint8_t>(nslot[0], 0), std::vector<uint8_t>(nslot[1], 0)};
    for (const LadderLaunch &ln : l.launches) walk(pl.tasks, pl.steps, pl.slots, ln, nslot, stored, n);
    for (const LadPair &p : pl.pairs) {
      need(p.pslot >= 0 && p.pslot < nslot[0] && stored[0][p.pslot], "prefix of pair", p.pslot);
      need(p.sslot >= 0 && p.sslot < nslot[1] && stored[1][p.sslot], "suffix of pair", p.sslot);
      need(p.leaf >= 0 && p.leaf < pl.nleaf, "leaf of pair", p.leaf);
    }
  }
  for (int32_t t : pl.term_leaf) need(t >= 0 && t < pl.nleaf, "leaf of term", t);
  for (int l = 0; l < LAD_LISTS; ++l) {
    check_grad(pl, l, n);
    steps += pl.lists[l].steps;
  }
  if (fault.empty()) return steps;
  std::snprintf(msg, size, "%s", fault.c_str());
  return -1;
}

extern "C" int check_ladder_pass(int B, unsigned long long state, unsigned long long budget) {
  return ladder_pass(B, state, budget);
}
