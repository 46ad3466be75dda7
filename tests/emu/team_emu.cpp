// The team PCG kernel (csrc/pcg_team.cu) with its own planner, run by the
// emulator of cta_emu.h on a chosen interleaving.  The test puts the kernel's
// source in team_kernel.inc (the inline PTX of its four helpers replaced by
// the functions below).  One scenario per run; prints "key value" lines.
#include <cuda_runtime.h>
#include "cta_emu.h"

#include <array>
#include <cmath>
#include <random>
#include <string>

static int g_smem_limit = 227 << 10;
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = g_smem_limit;
  return cudaSuccess;
}

namespace b200fem {
namespace {
inline void put_packet(double* slot, double v, unsigned half, unsigned tag) {
  unsigned* w = (unsigned*)(slot + 1);
  slot[0] = v;
  w[0] = half;
  w[1] = tag;
}
inline double get_packet(const double* slot, unsigned& half, unsigned& tag) {
  emu::yield();
  const unsigned* w = (const unsigned*)(slot + 1);
  half = w[0];
  tag = w[1];
  return slot[0];
}
inline unsigned long long team_ns() { return emu::M->clock_ns; }
inline void row_barrier() { emu::sync_named(480); }
}  // namespace
}  // namespace b200fem
using std::max;
using std::min;
#include "team_kernel.inc"

using namespace b200fem;

struct Problem {
  Engine eng;
  std::vector<int> rowptr{0}, col, diag, mirror;
  std::vector<double> S, divblk, kp, b, x, step, out;
  std::vector<float> Sf;
  bool dil = false;
  TeamHost th;
  // device-side arrays
  std::vector<unsigned char> stream;
  std::vector<double> row_pk, part_pk, t_pk;
  std::vector<unsigned> base;
  std::vector<int> g1, g2, act_node;
  unsigned long long ticket = 0;
  int flags[4] = {0, 0, 0, 0};
  TeamArgs a{};
};

// Models on nx x ny x nz grids, every node coupled to its 26 neighbours, stiff
// by `stiff` against the mass part (the iterations grow with it).
static void make(Problem& P, const std::vector<std::array<int, 3>>& grids, const std::vector<double>& stiff, double tol,
                 bool dil, unsigned seed) {
  std::mt19937 rng(seed);
  std::uniform_real_distribution<double> U(-1, 1);
  P.dil = dil;
  P.eng.row_off = {0};
  for (size_t m = 0; m < grids.size(); m++) {
    const auto [nx, ny, nz] = grids[m];
    const int r0 = P.eng.row_off.back(), n = nx * ny * nz;
    ModelDesc md;
    ModelHost mh;
    md.n_nodes = n;
    md.mat_kind = B200FEM_MAT_NEOHOOKEAN;
    md.mat_params[0] = 1000.0 * stiff[m];
    md.mat_params[1] = 0.3;
    for (int i = 0; i < n; i++) {
      mh.act_node.push_back(i);
      const int q[3] = {i % nx, i / nx % ny, i / nx / ny};
      for (int c = 0; c < 3; c++) md.rest.push_back(q[c] + 0.1 * U(rng));
      for (int j = 0; j < n; j++) {
        const int s[3] = {j % nx, j / nx % ny, j / nx / ny};
        if (std::abs(q[0] - s[0]) > 1 || std::abs(q[1] - s[1]) > 1 || std::abs(q[2] - s[2]) > 1) continue;
        if (i == j) P.diag.push_back((int)P.col.size());
        P.col.push_back(r0 + j);
      }
      P.rowptr.push_back((int)P.col.size());
    }
    mh.rest_vol.assign(1, (double)n);
    P.eng.models.push_back(md);
    P.eng.hosts.push_back(mh);
    P.eng.row_off.push_back(r0 + n);
  }
  const int R = P.eng.row_off.back(), M = (int)grids.size();
  P.S.assign(9 * P.col.size(), 0.0);
  P.mirror.assign(P.col.size(), 0);
  std::vector<int> model(R);
  for (int m = 0; m < M; m++)
    for (int r = P.eng.row_off[m]; r < P.eng.row_off[m + 1]; r++) model[r] = m;
  for (int r = 0; r < R; r++)
    for (int p = P.rowptr[r]; p < P.rowptr[r + 1]; p++) {
      const int j = P.col[p];
      int q = P.rowptr[j];
      while (P.col[q] != r) q++;
      P.mirror[p] = q;
      if (j <= r) continue;
      // -stiff w v v^T off the diagonal, the same added on both diagonals
      double v[3] = {U(rng), U(rng), U(rng)};
      for (int c = 0; c < 3; c++)
        for (int d = 0; d < 3; d++) {
          const double k = stiff[model[r]] * (v[c] * v[d] + (c == d ? 0.2 : 0.0));
          P.S[9 * (size_t)p + 3 * c + d] = -k;
          P.S[9 * (size_t)q + 3 * c + d] = -k;
          P.S[9 * (size_t)P.diag[r] + 3 * c + d] += k;
          P.S[9 * (size_t)P.diag[j] + 3 * c + d] += k;
        }
    }
  for (int r = 0; r < R; r++)
    for (int c = 0; c < 3; c++) P.S[9 * (size_t)P.diag[r] + 4 * c] += 1.0;
  P.divblk.resize(3 * P.col.size());
  for (double& v : P.divblk) v = 0.3 * U(rng);
  P.kp.resize(R);
  for (double& v : P.kp) v = 0.5 + 0.5 * U(rng);
  P.b.resize(3 * (size_t)R);
  for (double& v : P.b) v = U(rng);
  P.x.assign(3 * (size_t)R, 0.0);
  P.act_node.resize(R);
  std::iota(P.act_node.begin(), P.act_node.end(), 0);
  P.out.assign(4 * (size_t)M, -1.0);
  P.step.assign(8 * (size_t)M, 0.0);
  for (int m = 0; m < M; m++) {
    P.step[8 * m] = 1.0;  // h: c = h^2 + h beta = 1
    P.step[8 * m + 6] = tol;
  }
}
static bool plan(Problem& P, int grid_max, bool fp32) {
  P.eng.precision = fp32 ? B200FEM_PREC_MIXED : B200FEM_PREC_FP64;
  if (!plan_team(P.eng, grid_max, P.rowptr, P.col, P.diag, P.dil, P.th)) return false;
  const int R = P.eng.row_off.back();
  P.stream.assign((size_t)std::max(P.th.stream, 1) * P.th.step_bytes, 0);
  P.row_pk.assign(8 * (size_t)R, 0.0);
  P.t_pk.assign(4 * (size_t)R, 0.0);
  P.part_pk.assign(8 * P.th.slots.size(), 0.0);
  P.base.assign(P.eng.hosts.size(), 0u);
  P.Sf.assign(P.S.begin(), P.S.end());
  if (fp32) P.S.assign(P.Sf.begin(), P.Sf.end());
  P.g1.assign(P.th.blk.size(), -1);
  P.g2.assign(P.th.blk.size(), -1);
  for (size_t q = 0; q < P.th.blk.size(); q++)
    if (P.th.blk[q] >= 0) {
      P.g1[q] = P.th.blk[q];             // d_row's entry of col
      P.g2[q] = P.mirror[P.th.blk[q]];   // d_col's entry of row
    }
  TeamArgs& a = P.a;
  a.slots = P.th.slots.data();
  a.n_slots = (int)P.th.slots.size();
  a.ticket = &P.ticket;
  a.rows = P.th.rows.data();
  a.pub = P.th.pub.data();
  a.diag = P.th.diag.data();
  a.halo = P.th.halo.data();
  a.group = P.th.group.data();
  a.blk = P.th.blk.data();
  a.cl = P.th.cl.data();
  a.g1 = P.g1.data();
  a.g2 = P.g2.data();
  a.stream = P.stream.data();
  a.S = fp32 ? (const void*)P.Sf.data() : (const void*)P.S.data();
  a.b = P.b.data();
  a.x = P.x.data();
  a.step = P.step.data();
  a.model_out = P.out.data();
  a.flags = P.flags;
  a.timeout_ns = 1ull << 40;
  a.skip_cta = -1;
  a.max_iter = 20000;
  a.n_rows = R;
  a.base = P.base.data();
  a.row_pk = P.row_pk.data();
  a.part_pk = P.part_pk.data();
  a.t_pk = P.t_pk.data();
  a.act_node = P.act_node.data();
  a.divblk = P.divblk.data();
  a.node_kp = P.kp.data();
  return true;
}
static std::string launch(Problem& P, emu::Machine& m) {
  const bool fp32 = P.eng.precision == B200FEM_PREC_MIXED;
  const TeamArgs a = P.a;
  TeamKernel k = P.dil ? (fp32 ? team_kernel_of<float, true>(P.th.sets) : team_kernel_of<double, true>(P.th.sets))
                       : (fp32 ? team_kernel_of<float, false>(P.th.sets) : team_kernel_of<double, false>(P.th.sets));
  return emu::run(m, P.th.grid, kTeamThreads, P.th.smem, [a, k] { k(a); });
}
// largest relative residual over the models, in double
static double residual(const Problem& P) {
  const int R = P.eng.row_off.back();
  std::vector<double> y(3 * (size_t)R, 0.0), t(R, 0.0);
  for (int r = 0; r < R; r++)
    for (int p = P.rowptr[r]; p < P.rowptr[r + 1]; p++)
      for (int c = 0; c < 3; c++) {
        for (int d = 0; d < 3; d++) y[3 * r + c] += P.S[9 * (size_t)p + 3 * c + d] * P.x[3 * P.col[p] + d];
        t[r] += P.divblk[3 * (size_t)p + c] * P.x[3 * P.col[p] + c];
      }
  if (P.dil)
    for (int r = 0; r < R; r++)
      for (int p = P.rowptr[r]; p < P.rowptr[r + 1]; p++) {
        const int j = P.col[p];
        for (int c = 0; c < 3; c++) y[3 * r + c] += P.kp[j] * t[j] * P.divblk[3 * (size_t)P.mirror[p] + c];
      }
  double worst = 0;
  for (size_t m = 0; m + 1 < P.eng.row_off.size(); m++) {
    double rr = 0, bb = 0;
    for (int q = 3 * P.eng.row_off[m]; q < 3 * P.eng.row_off[m + 1]; q++) {
      rr += (P.b[q] - y[q]) * (P.b[q] - y[q]);
      bb += P.b[q] * P.b[q];
    }
    worst = std::max(worst, std::sqrt(rr / bb));
  }
  return worst;
}
static void report(const Problem& P, const std::string& hang) {
  printf("ended %s\nflag %d\n", hang.empty() ? "yes" : hang.c_str(), P.flags[0]);
  printf("residual %.17g\n", residual(P));
  double it = 0, conv = 1;
  for (size_t m = 0; 4 * m < P.out.size(); m++) {
    it = std::max(it, P.out[4 * m]);
    conv = std::min(conv, P.out[4 * m + 2]);
  }
  int stream = P.th.stream, mem = 0, kmax = 0;
  for (const TeamSlot& s : P.th.slots) {
    mem += s.steps_smem;
    kmax = std::max(kmax, s.k);
  }
  printf("iterations %g\nconverged %g\nsets %d\nslots %zu\nteam %d\ngrid %d\nstreamed %d\nkept %d\ntickets %llu\n", it, conv,
         P.th.sets, P.th.slots.size(), kmax, P.th.grid, stream, mem, P.ticket);
}

// ---- scenarios
// A solve: "solve <grids> <stiffness per model> <tol> <dil> <fp32> <CTAs> <smem KB> <variant>"
static int scenario_solve(char** v) {
  Problem P;
  std::vector<std::array<int, 3>> grids;
  std::vector<double> stiff;
  for (char* g = strtok(v[0], ";"); g; g = strtok(nullptr, ";")) {
    std::array<int, 3> q;
    if (sscanf(g, "%dx%dx%d", &q[0], &q[1], &q[2]) != 3) return 2;
    grids.push_back(q);
  }
  for (char* s = strtok(v[1], ";"); s; s = strtok(nullptr, ";")) stiff.push_back(atof(s));
  g_smem_limit = atoi(v[6]) << 10;
  make(P, grids, stiff, atof(v[2]), atoi(v[3]) != 0, 7);
  if (!plan(P, atoi(v[5]), atoi(v[4]) != 0)) {
    printf("ended not planned\n");
    return 0;
  }
  P.a.variant = atoi(v[7]);
  emu::Machine m;
  report(P, launch(P, m));
  return 0;
}

// An error is recorded (by a CTA of the same launch) just before warp `w` of a
// CTA that starts late reads the error word: "late_flag <w>"
static int scenario_late_flag(char** v) {
  const int w = atoi(v[0]);
  Problem P;
  make(P, {{3, 3, 3}}, {10.0}, 1e-8, false, 7);
  if (!plan(P, 1, false)) return 2;
  emu::Machine m;
  m.before = [&](emu::Fiber& f) {
    if (f.tid == 32 * w && !f.started) P.flags[0] = B200FEM_ERR_TIMEOUT;
  };
  report(P, launch(P, m));
  return 0;
}

// The true residual misses a tolerance one unit in the last place below it, so
// the solve restarts, and its squared form may already meet it; warp 14 is the
// last to read the verdict: "restart <seed>"
static int scenario_restart(char** v) {
  const unsigned seed = (unsigned)atoi(v[0]);
  double rel = 0;
  for (int run = 0; run < 2; run++) {
    Problem P;
    make(P, {{2, 1, 1}}, {1.0}, run ? std::nextafter(rel, 0.0) : 1e-12, false, seed);
    if (!plan(P, 1, false)) return 2;
    emu::Machine m;
    if (run) m.rank = [](const emu::Fiber& f) { return f.warp() == 14 ? 0 : 1; };
    const std::string hang = launch(P, m);
    rel = P.out[1];
    if (run) report(P, hang);
  }
  return 0;
}

// A team of two converges; another model's error is recorded then, CTA 1 is
// slow to go on and warp 14 of CTA 0 the last of its warps to look at the
// outcome of the iteration: "slow_warp <variant>"
static int scenario_slow_warp(char** v) {
  Problem P;
  make(P, {{6, 6, 6}}, {1.0}, 1e-6, false, 7);
  if (!plan(P, 2, false)) return 2;
  P.a.variant = atoi(v[0]);
  emu::Machine m;
  m.before = [&](emu::Fiber&) {
    auto& s = m.ctas[0]->shared["s_code"];
    if (P.flags[0] == 0 && !s.empty() && *(int*)(((uintptr_t)s.data() + 15) & ~(uintptr_t)15) != kRun)
      P.flags[0] = B200FEM_ERR_INVALID_ARG;
  };
  m.rank = [&](const emu::Fiber& f) {
    return P.flags[0] != 0 && (f.cta->block == 1 || f.warp() == 14) ? 0 : 1;
  };
  report(P, launch(P, m));
  return 0;
}

// Three models, three CTAs, a random interleaving; an error is recorded after
// `at` scheduling steps (0: never; -1: row 0 has a singular diagonal block, and
// its warp runs ahead).  A second solve follows, after an error
// with tickets, tags and packets cleared: "random <seed> <at> <variant> <dil>"
static int scenario_random(char** v) {
  Problem P;
  const unsigned seed = (unsigned)atoi(v[0]);
  const long at = atol(v[1]);
  make(P, {{9, 6, 5}, {3, 2, 2}, {4, 3, 3}}, {4.0, 1.0, 2.0}, 1e-6, atoi(v[3]) != 0, seed);
  if (!plan(P, 3, false)) return 2;
  P.a.variant = atoi(v[2]);
  const std::vector<double> S = P.S;
  size_t bad = 0;  // where row 0 lies among the slots' rows
  while (P.th.rows[bad] != 0) bad++;
  if (at < 0) {
    std::fill_n(&P.S[9 * (size_t)P.diag[0]], 9, 0.0);
    std::fill(P.kp.begin(), P.kp.begin() + P.eng.row_off[1], 0.0);
  }
  std::mt19937 rng(seed);
  emu::Machine m;
  // runs of one fiber's neighbours, then a jump: warps drift far apart
  m.choose = [&](size_t n) { return rng() % 8 ? 0 : rng() % n; };
  m.before = [&](emu::Fiber&) {
    if (at > 0 && (long)m.resumes >= at) P.flags[0] = B200FEM_ERR_INVALID_ARG;
  };
  if (at < 0)
    m.rank = [&](const emu::Fiber& f) {
      auto& s = f.cta->shared["s_slot"];
      if (s.empty() || m.resumes > 200000) return 1;  // (others poll for what this CTA publishes)
      const TeamSlot& sl = *(const TeamSlot*)(((uintptr_t)s.data() + 15) & ~(uintptr_t)15);
      if ((int)bad < sl.r0 || (int)bad >= sl.r0 + sl.nloc) return 1;
      return f.warp() == ((int)bad - sl.r0) % kSetRows / 10 ? 1 : 0;
    };
  report(P, launch(P, m));
  P.S = S;
  if (P.flags[0] != 0) {
    P.flags[0] = 0;
    P.ticket = 0;
    std::fill(P.base.begin(), P.base.end(), 0u);
    for (auto* v : {&P.row_pk, &P.part_pk, &P.t_pk}) std::fill(v->begin(), v->end(), 0.0);
  }
  for (size_t i = 0; i < P.b.size(); i++) {
    P.b[i] = -2 * P.b[i] + 0.1;
    P.x[i] = 0.01 * P.b[i];
  }
  emu::Machine m2;
  m2.choose = m.choose;
  const std::string hang = launch(P, m2);
  printf("again %s\nagain_flag %d\nagain_residual %.17g\n", hang.empty() ? "yes" : hang.c_str(), P.flags[0], residual(P));
  return 0;
}

// Two CTAs: the first members of a team of two wait until the other CTA ends a
// long solve of another model.  A scheduling step takes 10 ns, the limit of a
// wait is 1 ms: "queue"; "queue gone": the second member never publishes.
static int scenario_queue(bool gone) {
  Problem P;
  make(P, {{5, 4, 4}, {5, 4, 4}, {9, 6, 5}}, {100.0, 0.01, 1.0}, 1e-8, false, 7);
  P.eng.models[1].mat_params[0] = P.eng.models[0].mat_params[0] = 1e6;  // queued first
  if (!plan(P, 2, false)) return 2;
  P.a.timeout_ns = 1000000;
  emu::Machine m;
  if (gone)  // (its packets are lost)
    m.before = [&](emu::Fiber&) {
      for (const TeamSlot& s : P.th.slots)
        if (s.rank == 1) P.part_pk[4 * (s.s0 + 1) + 1] = P.part_pk[4 * (P.th.slots.size() + s.s0 + 1) + 1] = 0;
    };
  report(P, launch(P, m));
  printf("clock_us %llu\n", (unsigned long long)(m.clock_ns / 1000));
  return 0;
}

int main(int argc, char** argv) {
  const std::string s = argc > 1 ? argv[1] : "";
  if (s == "solve" && argc == 10) return scenario_solve(argv + 2);
  if (s == "late_flag" && argc == 3) return scenario_late_flag(argv + 2);
  if (s == "restart" && argc == 3) return scenario_restart(argv + 2);
  if (s == "slow_warp" && argc == 3) return scenario_slow_warp(argv + 2);
  if (s == "random" && argc == 6) return scenario_random(argv + 2);
  if (s == "queue") return scenario_queue(argc == 3);
  return 2;
}
