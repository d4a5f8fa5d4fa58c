// The host side of k_tail: which levels it takes, where their tables and vectors lie in shared memory, and
// the program of phases of a sub-cycle.  Host arithmetic alone, no CUDA, so that the programs can be checked
// without a GPU.  Mg is the hierarchy: lv[k].{n, W, Wq, gen, ap_ok, lmax}, opt, lc, pre_at(k), post_at(k).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <vector>

#include "dec_b200.h"

namespace decb {

constexpr int kTailBlock = 256;  // threads of the per-level kernels (TB): their sums are over blocks of rows
constexpr int kTailApW = 8;      // slots of a row of A P (kApW)
constexpr int kTailThreads = 384;
constexpr int kTailLevels = 12;
constexpr int kTailMaxCluster = 16;
// The most phases of a program (5 MB), and of all full-multigrid programs of a workspace together: cycle counts are
// unrolled, and beyond this they go level by level.  Twelve levels of V(3,3) with 5 W-cycles a level have 15,100.
constexpr size_t kTailMaxPhases = 1 << 16;
constexpr uint16_t kTailNone = 0xffff;     // a table's padding entry
constexpr size_t kTailSmem = 224 * 1024;   // vectors and tables per CTA; the rest of the 227 KB is static

enum TailType : uint8_t {
  TT_RESTRICT_G, TT_LOAD, TT_LOADX, TT_STORE, TT_ADDU, TT_ZERO, TT_SWEEP, TT_AP, TT_RESTRICT, TT_PROLONG,
  TT_COARSE, TT_CG  // from here on: phases that all threads of the CTA go through
};
// Buffers of a level.  Chebyshev / Jacobi: x, y (ping-pong, residual), b, d (correction form).
// CG: x, r, b, two p's, q, Δx.
enum TailBuf : uint8_t { TB_X = 0, TB_Y = 1, TB_B = 2, TB_D = 3, TB_P1 = 4, TB_Q = 5, TB_E = 6, TB_NBUF = 7 };
// What a sweep does with its residual (SweepMode and sweep_rows' PV); none: a Chebyshev step.
enum TailMode : uint8_t {
  TM_RESID = 1,
  TM_JACOBI = 2,
  TM_FROM_ZERO = 4,  // x = 0
  TM_PREV = 8,       // x_prev is what out holds (else 0)
  TM_PZ = 16,        // x_prev = P z
  TM_ADD = 32,       // out += the result
  TM_OLD = TM_PREV | TM_ADD
};

// One phase, every table and vector as a byte offset in dynamic shared memory (resolved on the host: the
// kernel reads five 16-byte words per phase instead of a level's descriptor).
struct alignas(16) TailOp {
  uint8_t type, mode, add, zero;     // mode: TailMode; add: prolong onto the iterate; zero: CG from x = 0
  uint8_t barrier;                   // starts with a cluster barrier (else __syncthreads)
  uint8_t split;                     // a dense product's rows / a restriction's rows are shared over the CTAs
  uint8_t rep;                       // the level is kept by every CTA
  uint8_t steps;                     // CG steps
  int n, chunk;                      // rows of the phase, rows per CTA
  uint32_t x, b, out, z;             // vectors: iterate / source, right-hand side, result, level + 1's
  uint32_t t0, t1, t2, t3;           // col, off, diag, 1/diag | apc, apv, diag, 1/diag | rself, ridx, rw
  uint32_t t4, t5;                   // parents pa, pb | CG: second p, q
  uint16_t W, level;                 // slots per row; level of the hierarchy's tail (host only)
  uint32_t t6;                       // CG: Δx
  double p0, p1;                     // c1, c2 (1/θ for a first step, ω for Jacobi)
};
constexpr int kTailOpWords = sizeof(TailOp) / 16;
static_assert(sizeof(TailOp) == 80, "five 16-byte words");

// One level; the t_* are byte offsets of its tables in dynamic shared memory (the CTA's own rows, row-major).
struct TailLevel {
  int n, W, Wq, chunk;               // chunk: rows per CTA (n where every CTA keeps the level)
  int rep, rchunk;                   // rep: kept by every CTA; rchunk: rows of level + 1 a CTA restricts
  uint32_t t_col, t_off, t_diag, t_dinv, t_pa, t_pb, t_apc, t_apv, t_rself, t_ridx, t_rw;
  uint32_t buf[TB_NBUF];             // byte offsets of the vectors
};

// How a workspace's cycles use the tail kernel (k_tail): levels lt .. last run in one launch on clusters
// of C CTAs, one per right-hand side.
struct TailPlan {
  bool on = false;
  int lt = 0, last = 0, C = 1, pfuse = 0, max_rows = 0;
  size_t smem = 0;                // dynamic shared memory: the tables, the vectors, the CG sums' block partials
  uint32_t image_bytes = 0, part = 0, part_len = 0;
  TailLevel lv[kTailLevels] = {};
};

// What a tail launch is entered for.
enum TailEntry {
  TE_CORRECT = 0,   // b_lt = R r of the level above; cycles with μ = the parameter (and μ - 1, ... 1); z out
  TE_CYCLE = 1,     // lt = 0: one cycle in place on FP64 panels
  TE_STEP = 2,      // lt = 0: inner_cycles cycles from zero; the result is stored (0) or added to u (1)
  TE_FMG = 3,       // full multigrid with `parameter` cycles a level, b restricted from the level above (lt > 0)
                    // or loaded (lt = 0)
};
inline int64_t tail_key(int entry, int param) { return (int64_t)entry << 32 | (uint32_t)param; }

// Does the level's program use A P (k_sweep_ap's form of the first post-smoothing step)?
template <class Mg>
bool tail_uses_ap(const Mg& mg, int l, int pfuse) {
  const int pre = mg.pre_at(l), post = mg.post_at(l);
  return mg.opt.smoother == DEC_SMOOTH_CHEBYSHEV && mg.lv[l].ap_ok && post >= 2 && pfuse != 0 &&
         (pre == 0 || (pfuse == 3 && post == 2));
}

// The largest coarsest level whose dense product every CTA computes whole (no cluster barrier).
constexpr int kTailDenseOwn = 100;
constexpr int kTailRows = 1536;  // rows of a level per CTA
constexpr int kTailRowsFew = 400;  // where a level has two phases of smoothing or fewer
// The largest level that every CTA keeps whole: its phase costs one SM's work on all rows instead of a
// cluster barrier and reads from other CTAs.  The smaller bound where that lets the clusters take one
// more level.
constexpr int kTailRep = 700, kTailRepSmall = 256;

// Emits the phases of mu_cycle / cg_mu_cycle / fmg_T, statement for statement.
template <class Mg>
struct TailBuilder {
  const Mg& mg;
  const TailPlan& cfg;
  std::vector<TailOp> ops;
  size_t most = kTailMaxPhases;
  bool full = false;  // more than `most` phases: the program is not usable

  bool cg() const { return mg.opt.smoother == DEC_SMOOTH_CG; }
  TailOp& emit(TailType t, int l) {
    const TailLevel& L = cfg.lv[l - cfg.lt];
    TailOp op{};
    op.type = t;
    op.level = (uint16_t)(l - cfg.lt);
    op.n = L.n;
    op.chunk = L.chunk;
    op.rep = (uint8_t)L.rep;
    op.W = (uint16_t)L.W;
    op.t0 = L.t_col;
    op.t1 = L.t_off;
    op.t2 = L.t_diag;
    op.t3 = L.t_dinv;
    op.t4 = L.t_pa;
    op.t5 = L.t_pb;
    op.b = buf(l, TB_B);
    full = full || ops.size() >= most;
    if (full && !ops.empty()) ops.pop_back();
    ops.push_back(op);
    return ops.back();
  }
  // a vector's offset; one that the layout has not reserved would be the tables'
  uint32_t buf(int l, int b) const {
    const uint32_t o = cfg.lv[l - cfg.lt].buf[b];
    if (o < cfg.image_bytes) throw std::logic_error("multigrid: a tail vector that its layout has not reserved");
    return o;
  }
  void interval(int l, double& theta, double& delta, double& sigma) const {
    const double hi = mg.lv[l].lmax, lo = hi / mg.opt.cheb_ratio;
    theta = (hi + lo) / 2;
    delta = (hi - lo) / 2;
    sigma = theta / delta;
  }
  void cheb_n(TailOp& op, int mode, double sigma, double delta, double& rho) const {
    const double rho_new = 1 / (2 * sigma - rho);
    op.mode = (uint8_t)mode;
    op.p0 = rho_new * rho;
    op.p1 = 2 * rho_new / delta;
    rho = rho_new;
  }
  TailOp& sweep(int l, int x, int b, int out) {
    TailOp& op = emit(TT_SWEEP, l);
    op.x = buf(l, x);
    op.b = buf(l, b);
    op.out = buf(l, out);
    return op;
  }
  int smooth(int l, int x, bool zero_x, int sweeps) {
    double theta, delta, sigma;
    interval(l, theta, delta, sigma);
    double rho = 1 / sigma;
    const bool from_zero = zero_x;
    int other = x == TB_X ? TB_Y : TB_X;
    for (int it = 0; it < sweeps; ++it) {
      TailOp& op = sweep(l, x, TB_B, other);
      if (mg.opt.smoother == DEC_SMOOTH_JACOBI) {
        op.mode = TM_JACOBI;
        op.p1 = mg.opt.omega;
      } else if (it == 0) {
        op.p1 = 1.0 / theta;
      } else {
        cheb_n(op, it == 1 && from_zero ? 0 : TM_PREV, sigma, delta, rho);
      }
      if (zero_x) op.mode |= TM_FROM_ZERO;
      std::swap(x, other);
      zero_x = false;
    }
    return x;
  }
  void ap(int l, int b, int out, int z, double theta) {
    TailOp& op = emit(TT_AP, l);
    const TailLevel& L = cfg.lv[l - cfg.lt];
    op.t0 = L.t_apc;
    op.t1 = L.t_apv;
    op.b = buf(l, b);
    op.out = buf(l, out);
    op.z = buf(l + 1, z);
    op.p0 = 1.0 / theta;
  }
  void restrict_to(int l, int src) {  // the phase's rows are level l + 1's
    const TailLevel &L = cfg.lv[l - cfg.lt], &Lc = cfg.lv[l + 1 - cfg.lt];
    TailOp& op = emit(TT_RESTRICT, l);
    op.n = Lc.n;
    op.chunk = L.rchunk;
    op.rep = (uint8_t)(L.rep && Lc.rep);
    op.split = (uint8_t)(Lc.rep && !L.rep);
    op.W = (uint16_t)L.Wq;
    op.t0 = L.t_rself;
    op.t1 = L.t_ridx;
    op.t2 = L.t_rw;
    op.x = buf(l, src);
    op.out = buf(l + 1, TB_B);
  }
  void prolong(int l, int x, int z, bool assign) {
    TailOp& op = emit(TT_PROLONG, l);
    op.out = buf(l, x);
    op.z = buf(l + 1, z);
    op.add = assign ? 0 : 1;
  }
  void zero(int l, int x) { emit(TT_ZERO, l).out = buf(l, x); }
  void cg_smooth(int l, bool zero_x, int steps) {
    if (steps == 0) return;
    TailOp& op = emit(TT_CG, l);
    op.steps = (uint8_t)steps;
    op.zero = zero_x ? 1 : 0;
    op.x = buf(l, TB_X);
    op.out = buf(l, TB_Y);
    op.z = buf(l, TB_D);
    op.t4 = buf(l, TB_P1);
    op.t5 = buf(l, TB_Q);
    op.t6 = buf(l, TB_E);
  }
  void residual(int l, int x, int out) { sweep(l, x, TB_B, out).mode = TM_RESID; }
  // the iterate of level l after one μ-cycle from buffer x (zero if zero_x)
  int cycle(int l, int x, bool zero_x, int mu) {
    if (full) return x;
    if (cg()) {
      cg_smooth(l, zero_x, mg.pre_at(l));
      if (mg.pre_at(l) > 0) zero_x = false;
      if (l >= cfg.last) {
        if (zero_x) zero(l, TB_X);
        return TB_X;
      }
      if (!zero_x) residual(l, TB_X, TB_Y);
      restrict_to(l, zero_x ? TB_B : TB_Y);
      int z = cycle(l + 1, TB_X, true, mu);
      if (mu > 1) z = cycle(l + 1, z, false, mu - 1);
      prolong(l, TB_X, z, zero_x);
      cg_smooth(l, false, mg.post_at(l));
      return TB_X;
    }
    if (l == mg.lc) {
      if (mg.opt.coarse_solver == 1) return smooth(l, x, zero_x, std::max(1, mg.pre_at(l) + mg.post_at(l)));
      TailOp& op = emit(TT_COARSE, l);
      op.split = cfg.C > 1 && mg.lv[l].n > kTailDenseOwn ? 1 : 0;
      op.out = buf(l, TB_X);
      return TB_X;
    }
    x = smooth(l, x, zero_x, mg.pre_at(l));
    zero_x = zero_x && mg.pre_at(l) == 0;
    int r = TB_B;
    if (!zero_x) {
      r = x == TB_X ? TB_Y : TB_X;
      residual(l, x, r);
    }
    restrict_to(l, r);
    int z = cycle(l + 1, TB_X, true, mu);
    if (mu > 1) z = cycle(l + 1, z, false, mu - 1);
    const int post = mg.post_at(l);
    double theta, delta, sigma;
    interval(l, theta, delta, sigma);
    double rho = 1 / sigma;
    if (mg.opt.smoother == DEC_SMOOTH_CHEBYSHEV && post >= 2 && mg.lv[l].ap_ok) {
      if (zero_x && cfg.pfuse != 0) {  // smooth_prolonged
        int other = x == TB_X ? TB_Y : TB_X;
        ap(l, TB_B, other, z, theta);
        std::swap(x, other);
        for (int it = 1; it < post; ++it) {
          TailOp& op = sweep(l, x, TB_B, other);
          cheb_n(op, it == 1 ? TM_PZ : TM_PREV, sigma, delta, rho);
          if (it == 1) op.z = buf(l + 1, z);
          std::swap(x, other);
        }
        return x;
      }
      if (!zero_x && cfg.pfuse == 3 && post == 2) {  // smooth_correction
        ap(l, r, TB_D, z, theta);
        TailOp& op = sweep(l, TB_D, r, x);
        cheb_n(op, TM_PZ | TM_ADD, sigma, delta, rho);
        op.z = buf(l + 1, z);
        return x;
      }
    }
    prolong(l, x, z, zero_x);
    return smooth(l, x, false, post);
  }
  int fmg(int l, int cycles) {
    int z = TB_X;
    bool zero = true;
    if (l < cfg.last) {
      restrict_to(l, TB_B);
      const int zc = fmg(l + 1, cycles);
      prolong(l, z, zc, true);
      zero = false;
    }
    for (int c = 0; c < cycles && !full; ++c) {
      z = cycle(l, z, zero, mg.opt.mu);
      zero = false;
    }
    if (zero) this->zero(l, z);
    return z;
  }
  // false: too many phases
  bool build(int entry, int param) {
    const int lt = cfg.lt;
    int z = TB_X;
    if (lt > 0) {
      emit(TT_RESTRICT_G, lt).out = buf(lt, TB_B);
    } else {
      emit(TT_LOAD, lt).out = buf(lt, TB_B);
      if (entry == TE_CYCLE) emit(TT_LOADX, lt).out = buf(lt, TB_X);
    }
    if (entry == TE_CORRECT) {
      z = cycle(lt, z, true, param);
      if (param > 1) z = cycle(lt, z, false, param - 1);
    } else if (entry == TE_CYCLE) {
      z = cycle(lt, z, false, mg.opt.mu);
    } else if (entry == TE_STEP) {
      for (int c = 0; c < mg.opt.inner_cycles; ++c) z = cycle(lt, z, c == 0, mg.opt.mu);
    } else {
      z = fmg(lt, param);
    }
    emit(entry == TE_STEP && param ? TT_ADDU : TT_STORE, lt).x = buf(lt, z);
    if (cfg.C > 1 && !full) barriers();
    return !full;
  }
  // Which phases start with a cluster barrier.  Rows of a split level are written by their CTA alone and
  // read by others through `gather`; a level that every CTA keeps is written by each, or pushed to all.
  // A phase needs the barrier when it reads what others may have written since the last one, writes what
  // they may still read, follows a push, or pushes (the targets may still be read).  The first access to
  // another CTA's memory waits for all CTAs to run: a CG from zero reads none, but its sums store to all.
  void barriers() {
    bool wrote = true, read = false, pushed = false, running = false;
    for (TailOp& op : ops) {
      const bool split = !cfg.lv[op.level].rep;
      const bool csplit = op.level + 1 < kTailLevels && cfg.lv[op.level + 1].n > 0 && !cfg.lv[op.level + 1].rep;
      bool reads = false, writes = false, pushes = false;
      switch (op.type) {
        case TT_RESTRICT_G: case TT_LOAD: case TT_LOADX: case TT_ZERO: writes = split; break;
        case TT_SWEEP:
          reads = (split && !(op.mode & TM_FROM_ZERO)) || (csplit && (op.mode & TM_PZ));
          writes = split;
          break;
        case TT_AP: case TT_PROLONG: reads = csplit; writes = split; break;
        case TT_RESTRICT:
          reads = split;
          writes = csplit;
          pushes = split && !csplit;
          break;
        case TT_COARSE: pushes = op.split != 0; break;
        case TT_CG: reads = split && !op.zero; writes = split; break;
        default: break;  // TT_STORE, TT_ADDU: the CTA's own rows
      }
      const bool sums = op.type == TT_CG && split;
      op.barrier = ((reads && wrote) || (writes && read) || pushed || pushes || (sums && !running)) ? 1 : 0;
      if (op.barrier) wrote = read = pushed = false;
      running |= op.barrier != 0;
      read |= reads;
      wrote |= writes;
      pushed |= pushes;
      if (sums) {  // its sums' barriers; x += Δx comes after the last
        read = false;
        wrote = !op.zero;
      }
    }
  }
};

// The tables and vectors of levels lt .. last at cluster size c.C; false if they do not fit.
template <class Mg>
bool tail_layout(const Mg& mg, TailPlan& c, size_t es, int K, int rep_rows) {
  const bool cg = mg.opt.smoother == DEC_SMOOTH_CG, dense = !cg && mg.opt.coarse_solver != 1;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 15) / 16 * 16;
    return (uint32_t)o;
  };
  for (auto& l : c.lv) l = TailLevel{};
  for (int k = c.lt; k <= c.last; ++k) {
    TailLevel& t = c.lv[k - c.lt];
    const auto& L = mg.lv[k];
    t.n = L.n;
    t.W = L.W;
    t.Wq = L.Wq;
    t.rep = c.C == 1 || L.n <= rep_rows;
    t.chunk = t.rep ? L.n : (L.n + c.C - 1) / c.C;
    const int rb = kTailBlock / K;  // rows of a block of the sums
    if (cg && !t.rep) t.chunk = (t.chunk + rb - 1) / rb * rb;
    if (t.chunk > c.max_rows) return false;
  }
  for (int k = c.lt; k <= c.last; ++k) {
    TailLevel& t = c.lv[k - c.lt];
    const size_t rows = t.chunk;
    if (k < c.last || !dense) {
      t.t_col = take(rows * t.W * 2);
      t.t_off = take(rows * t.W * es);
    }
    t.t_diag = take(rows * es);
    if (!cg) t.t_dinv = take(rows * es);
    if (k == c.last) break;
    const TailLevel& tc = c.lv[k + 1 - c.lt];
    t.t_pa = take(rows * 2);
    t.t_pb = take(rows * 2);
    if (tail_uses_ap(mg, k, c.pfuse)) {
      t.t_apc = take(rows * kTailApW * 2);
      t.t_apv = take(rows * kTailApW * es);
    }
    t.rchunk = tc.rep && t.rep ? tc.n : (tc.n + c.C - 1) / c.C;
    if (!tc.rep) t.rchunk = tc.chunk;
    t.t_rself = take((size_t)t.rchunk * 2);
    t.t_ridx = take((size_t)t.rchunk * t.Wq * 2);
    t.t_rw = take((size_t)t.rchunk * 2 * es);
  }
  c.image_bytes = (uint32_t)at;
  for (int k = c.lt; k <= c.last; ++k) {
    // TB_D: a cycle entered with an iterate may end in the correction form (W-cycles, cycles after a first
    // one, and on every level full multigrid, which prolongs before it cycles)
    const int nb = cg ? TB_NBUF : mg.opt.smoother == DEC_SMOOTH_CHEBYSHEV && mg.post_at(k) == 2 ? 4 : 3;
    for (int b = 0; b < nb; ++b) c.lv[k - c.lt].buf[b] = take((size_t)c.lv[k - c.lt].chunk * es);
  }
  if (cg) {
    c.part_len = (uint32_t)((c.lv[0].n + kTailBlock / K - 1) / (kTailBlock / K));
    c.part = take((size_t)c.part_len * 16);
  }
  c.smem = at;
  return at <= kTailSmem;
}

// Which levels run in k_tail, and on what clusters: the largest clusters (up to 16 CTAs) of which the
// device holds one per right-hand side at a time, and from the coarsest level up as many levels as their
// shared memory takes.  Only while a right-hand side gets a cluster of kTailMinCluster CTAs (7 of 16, or
// 15 of 8): with more right-hand sides the per-level kernels carry enough rows that a launch is no longer
// all latency (32 FP32 right-hand sides, four to a cluster: 0.6-0.86 of the per-level kernels' speed).
// Measured without / with (us): icosphere L6, V(3,3), FP64: 662 / 470 (1 right-hand side), 842 / 644 (8);
// L4: 435 / 288, 510 / 298; CG V-cycles on L6: 1,292 / 674, W-cycles 4,462 / 1,652.  A V(0,2)-cycle is
// three phases a level: levels of more than kTailRowsFew rows per CTA stay outside (L6, FP32, 8 right-hand
// sides: 391 / 378, with L5 inside 395 / 422), and few FP32 right-hand sides altogether (1: 292 / 301;
// 4: 377 / 351).  In FP32 over a dense coarsest level of more than kTailDenseFew vertices, V(0,2) stays outside
// with more than 4 right-hand sides and W(0,2) with fewer than 4: a 65 x 65 grid over 9 x 9 V(0,2) 352 / 365 (8;
// with 4 352 / 305), 257 x 257 over 9 x 9 W(0,2) 1,118 / 1,211 (1; 0.90 of it with 4), 129 x 97 over 17 x 13
// 553 / 576 (1; 0.85 with 4); over 5 x 4 0.87 and 0.69 in their place, in FP64 between 0.99 and 1.01, and less.
constexpr int kTailMinCluster = 8;
constexpr int kTailDenseFew = 64;
// K, npanels: the panels' width and count; prec: 0 FP64, 1 FP32; pfuse: the fused prolongation's mode;
// held(C): how many clusters of C CTAs the device holds at a time.
template <class Mg, class Held>
void tail_decide(const Mg& mg, TailPlan& c, int K, int npanels, int prec, int pfuse, Held held) {
  const dec_mg_options& o = mg.opt;
  const bool cg = o.smoother == DEC_SMOOTH_CG;
  if (o.smoother == DEC_SMOOTH_LEARNED || prec == 2 || mg.lv.size() < 2) return;
  if (!cg && o.coarse_solver == 2) return;  // a shift per right-hand side
  c.pfuse = pfuse;
  c.last = cg ? (int)mg.lv.size() - 1 : mg.lc;
  if (c.pfuse == 2 || c.last == 0) return;
  if (!cg && o.coarse_solver == 0 && mg.lv[c.last].n > kTailRepSmall) return;
  if (cg && K > 8) return;  // the sums take blocks of 32 rows at least (a guard: 16 groups get no clusters of 8 here)
  const int groups = K * npanels;
  const size_t es = prec == 1 ? 4 : 8;
  for (c.C = kTailMaxCluster; c.C > 1 && held(c.C) < groups;) c.C /= 2;
  if (c.C < kTailMinCluster) return;
  const int sweeps = mg.pre_at(c.last - 1) + mg.post_at(c.last - 1);
  const bool few = !cg && o.mu == 1 && sweeps <= 2;
  if (few && prec == 1 && groups < 4) return;
  if (prec == 1 && o.coarse_solver == 0 && mg.pre_at(c.last - 1) == 0 && sweeps <= 2 && mg.lv[c.last].n > kTailDenseFew &&
      (o.mu == 1 ? groups > 4 : groups < 4))
    return;
  c.max_rows = few ? kTailRowsFew : kTailRows;
  auto fits = [&](int lt, int rep_rows) {
    c.lt = lt;
    return c.last - lt < kTailLevels && !mg.lv[lt].gen && tail_layout(mg, c, es, K, rep_rows);
  };
  auto finest = [&](int rep_rows) {
    int lt = c.last + 1;
    while (lt > 0 && fits(lt - 1, rep_rows)) --lt;
    return lt;
  };
  const int lt_small = finest(kTailRepSmall), lt_big = finest(kTailRep);
  const int rep_rows = lt_small < lt_big ? kTailRepSmall : kTailRep, lt = std::min(lt_small, lt_big);
  if (lt > c.last || (lt > 0 && mg.lv[lt - 1].gen)) return;
  if (mg.lv[lt].n <= rep_rows) c.C = 1;  // nothing to split
  c.on = fits(lt, rep_rows);
}

}  // namespace decb
