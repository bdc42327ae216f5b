// Host check of the pipelined band sweep's plan
// (meshcfd_gb300/csrc/mcfd_pipeline_plan.h): executes it as k_lusgs_pipeline
// does -- every band its own steps in order, own rows through the ring, other
// bands' rows through single-use slots that start empty -- with the bands
// interleaved at random, and compares with the natural-order substitution bit
// for bit.  A band whose step reads an empty slot waits; a round in which no
// band advances is a deadlock.
//
// usage: pipeline_plan_check SEED -> "cases=<n> planned=<n> failures=<n>"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <set>

#include "../meshcfd_gb300/csrc/mcfd_pipeline_plan.h"

using namespace mcfd;

struct Sweep {
  std::vector<int> level_ptr, pos_cell, ent_ptr, ent_pos, ent_cell;
  std::vector<double> val;
};

// Levels of the substitution over adj (forward: lower columns, backward: higher), sorted by (level, cell)
static Sweep make_sweep(const std::vector<std::set<int>>& adj, bool forward, std::mt19937_64& rng) {
  const int C = (int)adj.size();
  std::vector<int> lev(C, 0);
  int nlev = 0;
  for (int s = 0; s < C; ++s) {
    const int i = forward ? s : C - 1 - s;
    for (int j : adj[i])
      if (forward ? j < i : j > i) lev[i] = std::max(lev[i], lev[j] + 1);
    nlev = std::max(nlev, lev[i] + 1);
  }
  Sweep S;
  S.level_ptr.assign(nlev + 1, 0);
  for (int i = 0; i < C; ++i) S.level_ptr[lev[i] + 1]++;
  for (int l = 0; l < nlev; ++l) S.level_ptr[l + 1] += S.level_ptr[l];
  std::vector<int> fill(S.level_ptr.begin(), S.level_ptr.end() - 1), pos(C);
  S.pos_cell.resize(C);
  for (int i = 0; i < C; ++i) {
    pos[i] = fill[lev[i]]++;
    S.pos_cell[pos[i]] = i;
  }
  std::uniform_real_distribution<double> u(-0.4, 0.4);
  S.ent_ptr.assign(1, 0);
  for (int p = 0; p < C; ++p) {
    const int i = S.pos_cell[p];
    for (int j : adj[i])
      if (forward ? j < i : j > i) {
        S.ent_pos.push_back(pos[j]);
        S.ent_cell.push_back(j);
        S.val.push_back(u(rng));
      }
    S.ent_ptr.push_back((int)S.ent_pos.size());
  }
  return S;
}

static bool run(const Sweep& S, const PipelinePlanHost& H, const PipelineLimits& lim, const std::vector<double>& rhs,
                const std::vector<double>& diag, const std::vector<double>& ref, std::mt19937_64& rng) {
  const double empty = std::numeric_limits<double>::quiet_NaN();
  std::vector<std::vector<double>> sl(H.nc, std::vector<double>(lim.ring + lim.externals, empty));
  std::vector<double> out(rhs.size(), empty);
  std::vector<int> at(H.nc, 0);
  size_t written = 0;
  bool moved = true;
  while (moved) {
    moved = false;
    for (int turn = 0; turn < 4 * H.nc; ++turn) {
      const int k = (int)(rng() % H.nc);
      const int n_steps = H.step0[k + 1] - H.step0[k] - 1;
      if (at[k] >= n_steps) continue;
      const int* st = H.steps.data() + H.step0[k] + at[k];
      const int f = st[0] & 0xffffff, e = st[1] & 0xffffff, most = st[0] >> 24;
      if (e - f < 1 || e - f > H.max_step) return false;
      bool wait = false;
      std::vector<double> res(e - f);
      for (int r = f; r < e && !wait; ++r) {
        const size_t i = (size_t)H.chunk0[k] * kPipeChunk + r;
        const int p = H.pos[i], n = H.count[i];
        if (p < 0 || n > most || S.pos_cell[p] != H.cell[i] || H.row_of_cell[H.cell[i]] != (int)i) return false;
        double acc = rhs[H.cell[i]];
        for (int q = 0; q < n; ++q) {
          const unsigned slot = H.slots[4 * i + q];
          const double x = sl[k][slot & 0x7fff];
          if (slot & 0x8000) {
            if (x != x) {
              wait = true;
              break;
            }
          }
          acc = acc - S.val[S.ent_ptr[p] + q] * x;
        }
        res[r - f] = acc / diag[H.cell[i]];
      }
      if (wait) continue;
      for (int r = f; r < e; ++r) {
        const size_t i = (size_t)H.chunk0[k] * kPipeChunk + r;
        sl[k][r & (lim.ring - 1)] = res[r - f];
        for (int d = 0; d < 4; ++d)
          if (H.dest[4 * i + d] >= 0) {
            const int b = H.dest[4 * i + d] >> 16, slot = H.dest[4 * i + d] & 0xffff;
            if (b < 0 || b >= H.nc || slot < lim.ring || slot >= lim.ring + H.externals[b]) return false;
            if (sl[b][slot] == sl[b][slot]) return false;  // written twice
            sl[b][slot] = res[r - f];
          }
        out[H.cell[i]] = res[r - f];
        ++written;
      }
      ++at[k];
      moved = true;
    }
    if (!moved)  // no lucky draw: one pass over every band
      for (int k = 0; k < H.nc; ++k)
        if (at[k] < H.step0[k + 1] - H.step0[k] - 1) {
          // an unfinished band: the draws may have missed it; try again unless all are stuck
          moved = true;
          break;
        }
    static thread_local long rounds = 0;
    if (++rounds > 40000000) return false;  // deadlock
  }
  if (written != rhs.size()) return false;
  return std::memcmp(out.data(), ref.data(), out.size() * sizeof(double)) == 0;
}

int main(int argc, char** argv) {
  std::mt19937_64 rng(argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  long cases = 0, planned = 0, failures = 0;
  for (int rep = 0; rep < 60; ++rep) {
    const int nx = 1 + (int)(rng() % 40), ny = 1 + (int)(rng() % 40), C = nx * ny;
    std::vector<std::set<int>> adj(C);
    auto link = [&](int a, int b) {
      if (a != b && adj[a].size() < 4 && adj[b].size() < 4) adj[a].insert(b), adj[b].insert(a);
    };
    std::vector<int> id(C);
    for (int i = 0; i < C; ++i) id[i] = i;
    if (rep % 3 == 2) std::shuffle(id.begin(), id.end(), rng);
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        if (i + 1 < nx) link(id[j * nx + i], id[j * nx + i + 1]);
        if (j + 1 < ny && (rep % 4 != 1 || (i + j) % 2)) link(id[j * nx + i], id[(j + 1) * nx + i]);
      }
    if (rep % 3 == 1)
      for (int e = 0; e < C / 8; ++e) link((int)(rng() % C), (int)(rng() % C));
    for (bool forward : {true, false}) {
      const Sweep S = make_sweep(adj, forward, rng);
      std::vector<double> rhs(C), diag(C), ref(C);
      std::uniform_real_distribution<double> u(0.5, 1.5);
      for (int i = 0; i < C; ++i) rhs[i] = u(rng), diag[i] = u(rng);
      std::vector<int> pos(C);
      for (int p = 0; p < C; ++p) pos[S.pos_cell[p]] = p;
      for (int s = 0; s < C; ++s) {
        const int i = forward ? s : C - 1 - s, p = pos[i];
        double acc = rhs[i];
        for (int q = S.ent_ptr[p]; q < S.ent_ptr[p + 1]; ++q) acc = acc - S.val[q] * ref[S.ent_cell[q]];
        ref[i] = acc / diag[i];
      }
      const PipelineLimits limits[] = {{2048, 2048, 6000}, {64, 128, 200}, {16, 16, 40}};
      for (const PipelineLimits& lim : limits)
        for (int nc : {8, 16})
          for (int step : {16, 32}) {
            ++cases;
            PipelinePlanHost H;
            if (!plan_pipeline_host(S.level_ptr, S.pos_cell, S.ent_ptr, S.ent_pos, C, nc, step, lim, H)) continue;
            ++planned;
            if (!run(S, H, lim, rhs, diag, ref, rng)) ++failures;
          }
    }
  }
  std::printf("cases=%ld planned=%ld failures=%ld\n", cases, planned, failures);
  return failures ? 1 : 0;
}
