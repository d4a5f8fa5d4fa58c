// Checks the programs that csrc/mg_tail_plan.h plans for k_tail, on the host: every vector that a phase names
// is one that the layout reserved, and no CTA of a cluster reaches another's shared memory before that one is
// known to run, reads what another may still write, or writes what another may still read.
//
// One hierarchy and entry per line of standard input:
//   smoother precision pre post mu inner coarse_solver lc K npanels pfuse cycles levels (n W Wq ap_ok)*
// finest level first; answers with "off", or "on <first level> <CTAs> <phases>", "refused" behind it if a program
// would be too long, and a "fault ..." line for each violation.
#include <cstdio>
#include <iostream>
#include <map>
#include <set>
#include <sstream>
#include <string>

#include "mg_tail_plan.h"

using namespace decb;

struct Lv {
  int n, W, Wq;
  bool ap_ok, gen = false;
  double lmax = 2.0;
};
struct Hierarchy {
  dec_mg_options opt{};
  std::vector<Lv> lv;
  int lc = 0;
  int pre_at(int) const { return opt.pre; }
  int post_at(int) const { return opt.post; }
};

struct Replay {
  const Hierarchy& mg;
  const TailPlan& c;
  size_t es;
  std::string name;
  std::set<std::string> faults;
  // cluster barriers so far; when a vector (by byte offset) was last written by its owner, read or written by
  // its owner (local), read by another CTA, written by another CTA
  int epoch = 0;
  std::map<uint32_t, int> wrote, local, far_read, pushed;

  static int when(const std::map<uint32_t, int>& m, uint32_t v) {
    auto it = m.find(v);
    return it == m.end() ? -1 : it->second;
  }
  void fault(const std::string& s) { faults.insert(name + ": " + s); }
  static std::string at(const TailOp& op) { return " (type " + std::to_string(op.type) + ", level " + std::to_string(op.level) + ")"; }

  // the vector at this offset is one of level k's
  bool known(int k, uint32_t v) const {
    for (uint32_t b : c.lv[k].buf)
      if (b == v && v >= c.image_bytes) return true;
    return false;
  }
  void need(const TailOp& op, int k, uint32_t v) {
    if (!known(k, v)) fault("a vector that the layout has not reserved" + at(op));
  }
  void remote(const TailOp& op) {
    if (epoch == 0) fault("another CTA's memory before the first cluster barrier" + at(op));
  }
  void read(const TailOp& op, uint32_t v) {
    if (when(pushed, v) == epoch) fault("reads what another CTA writes" + at(op));
    local[v] = epoch;
  }
  void read_far(const TailOp& op, uint32_t v) {
    remote(op);
    if (when(wrote, v) == epoch) fault("reads what its owner may still write" + at(op));
    far_read[v] = epoch;
  }
  void write(const TailOp& op, uint32_t v) {
    if (when(far_read, v) == epoch || when(pushed, v) == epoch) fault("writes what another CTA may use" + at(op));
    wrote[v] = local[v] = epoch;
  }
  void push(const TailOp& op, uint32_t v) {
    remote(op);
    if (when(local, v) == epoch) fault("writes another CTA's vector in use" + at(op));
    pushed[v] = epoch;
  }

  void level_read(const TailOp& op, int k, uint32_t v, bool neighbours) {
    need(op, k, v);
    read(op, v);
    if (neighbours && !c.lv[k].rep) read_far(op, v);
  }
  void level_write(const TailOp& op, int k, uint32_t v) {
    need(op, k, v);
    write(op, v);
  }

  int parity = 0;
  void sums(const TailOp& op, bool own) {
    const uint32_t set = c.part + (uint32_t)parity * c.part_len * 8u;
    if (c.part < c.image_bytes || c.part + (size_t)c.part_len * 16 > c.smem) fault("the sums' partials out of the layout");
    parity ^= 1;
    if (own) {
      write(op, set);
    } else {
      push(op, set);
      ++epoch;
    }
    read(op, set);
  }
  // steps taken: as the data would have it
  void cg(const TailOp& op, int taken, bool curvature) {
    const int k = op.level;
    const bool own = c.C == 1 || c.lv[k].rep;
    const uint32_t x = op.x, r = op.out, q = op.t5, e = op.zero ? op.x : op.t6;
    uint32_t p = op.z, pn = op.t4;
    for (uint32_t v : {x, r, q, e, p, pn, op.b}) need(op, k, v);
    if (op.steps != mg.opt.pre && op.steps != mg.opt.post) fault("CG steps");
    read(op, op.b);
    if (!op.zero) level_read(op, k, x, true);
    write(op, r);
    write(op, e);
    sums(op, own);
    for (int it = 0; it < taken; ++it) {
      level_read(op, k, r, true);
      if (it) level_read(op, k, p, true);
      write(op, q);
      write(op, pn);
      sums(op, own);
      if (curvature && it + 1 == taken) break;
      write(op, e);
      write(op, r);
      sums(op, own);
      std::swap(p, pn);
    }
    if (!op.zero) write(op, x);
  }

  void run(const std::vector<TailOp>& ops, unsigned seed) {
    epoch = parity = 0;
    wrote.clear();
    local.clear();
    far_read.clear();
    pushed.clear();
    for (const TailOp& op : ops) {
      if (c.C > 1 && op.barrier) ++epoch;
      const int k = op.level;
      const bool split = !c.lv[k].rep;
      seed = seed * 1664525u + 1013904223u;
      switch (op.type) {
        case TT_RESTRICT_G: case TT_LOAD: case TT_LOADX: case TT_ZERO: level_write(op, k, op.out); break;
        case TT_STORE: case TT_ADDU: level_read(op, k, op.x, false); break;
        case TT_SWEEP:
          level_read(op, k, op.b, false);
          if (!(op.mode & TM_FROM_ZERO)) {
            level_read(op, k, op.x, true);
            if (op.x == op.out) fault("a sweep in place");
          }
          if (op.mode & TM_PZ) level_read(op, k + 1, op.z, true);
          level_write(op, k, op.out);
          break;
        case TT_AP:
          if (c.lv[k].t_apv == 0) fault("no A P table" + at(op));
          level_read(op, k, op.b, false);
          level_read(op, k + 1, op.z, true);
          level_write(op, k, op.out);
          break;
        case TT_PROLONG:
          level_read(op, k + 1, op.z, true);
          level_write(op, k, op.out);
          break;
        case TT_RESTRICT:
          level_read(op, k, op.x, true);
          if (split && c.lv[k + 1].rep) {
            need(op, k + 1, op.out);
            push(op, op.out);
          } else {
            level_write(op, k + 1, op.out);
          }
          break;
        case TT_COARSE:
          level_read(op, k, op.b, false);
          need(op, k, op.out);
          if (op.split) push(op, op.out);
          else write(op, op.out);
          break;
        case TT_CG: cg(op, (int)(seed >> 16) % (op.steps + 1), (seed >> 8 & 3) == 0); break;
        default: fault("an unknown phase");
      }
      (void)split;
    }
  }

  // tables first, then vectors that do not overlap
  void layout() {
    std::map<uint32_t, uint32_t> used;
    for (int k = 0; k <= c.last - c.lt; ++k)
      for (uint32_t b : c.lv[k].buf)
        if (b) used[b] = std::max(used[b], b + (uint32_t)(c.lv[k].chunk * es));
    uint32_t end = c.image_bytes;
    for (auto& u : used) {
      if (u.first < end) fault("vectors overlap");
      end = u.second;
    }
    if (end > c.smem || c.smem > kTailSmem) fault("shared memory exceeded");
  }
};

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    Hierarchy mg;
    int precision, K, npanels, pfuse, cycles, levels;
    in >> mg.opt.smoother >> precision >> mg.opt.pre >> mg.opt.post >> mg.opt.mu >> mg.opt.inner_cycles >>
        mg.opt.coarse_solver >> mg.lc >> K >> npanels >> pfuse >> cycles >> levels;
    mg.opt.cheb_ratio = 4.0;
    mg.opt.omega = 0.8;
    for (int k = 0; k < levels; ++k) {
      Lv l;
      int ap;
      in >> l.n >> l.W >> l.Wq >> ap;
      l.ap_ok = ap != 0;
      mg.lv.push_back(l);
    }
    TailPlan plan;
    // how many clusters of 2, 4, 8 and 16 CTAs of this size a B200 holds
    auto held = [](int C) { return C == 16 ? 7 : C == 8 ? 15 : C == 4 ? 33 : C == 2 ? 74 : 1 << 20; };
    tail_decide(mg, plan, K, npanels, precision, pfuse, held);
    if (!plan.on) {
      std::puts("off");
      continue;
    }
    std::vector<std::pair<int, int>> entries = {{TE_FMG, cycles}};
    if (plan.lt > 0) {
      for (int mu = 1; mu <= mg.opt.mu; ++mu) entries.push_back({TE_CORRECT, mu});
    } else {
      for (auto e : {std::pair<int, int>{TE_CYCLE, 0}, {TE_STEP, 0}, {TE_STEP, 1}}) entries.push_back(e);
    }
    if (tail_key(TE_FMG, cycles) == tail_key(TE_FMG, cycles + (1 << 16))) std::puts("fault two cycle counts, one key");
    size_t phases = 0;
    bool refused = false;
    std::set<std::string> faults;
    for (auto& e : entries) {
      Replay ck{mg, plan, precision == 1 ? 4u : 8u, "entry " + std::to_string(e.first) + "/" + std::to_string(e.second), {}};
      ck.layout();
      TailBuilder<Hierarchy> b{mg, plan, {}};
      if (!b.build(e.first, e.second)) {
        refused = true;
        continue;
      }
      if (b.ops.size() > kTailMaxPhases) faults.insert("a program of more than kTailMaxPhases phases");
      phases += b.ops.size();
      for (unsigned seed = 1; seed <= (mg.opt.smoother == DEC_SMOOTH_CG ? 12u : 1u); ++seed) ck.run(b.ops, seed);
      faults.insert(ck.faults.begin(), ck.faults.end());
    }
    std::printf("on %d %d %zu%s\n", plan.lt, plan.C, phases, refused ? " refused" : "");
    for (auto& f : faults) std::printf("fault %s\n", f.c_str());
  }
}
