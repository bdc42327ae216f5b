// Host planner of the pipelined band LU-SGS sweep (k_lusgs_pipeline in
// mcfd_pipeline.cu), plain C++ so that it also compiles without CUDA.
//
// Input: one sweep's rows in sweep order (positions, level by level) and each
// row's entries (column positions, in the row's entry order).  Block k of an
// nc-block cluster owns the cells [k * band_rows, (k + 1) * band_rows) and
// solves their rows in position order.  A triangular solve in natural cell
// order only ever reads lower columns (forward) or higher ones (backward), so
// the bands depend on one another in one direction and any order that keeps
// each band's own order ends.  The plan lists, per band:
//   steps: runs of at most max_step rows of one level (rows of a step are
//     independent), each as first row | most entries of a row << 24, then the
//     row count;
//   rows in chunks of kPipeChunk (padded): position (-1: padding), cell,
//     entry count, the shared-memory slot of each entry (own rows in a ring
//     of `ring` slots, rows of other bands in one slot each above it, bit 15
//     set), and up to four destinations (band << 16 | slot) of its solution;
//   externals: how many slots above the ring it receives.
// A sweep is not planned (ok stays false) where a row has more than four
// entries or destinations, an own row is read after the ring may have
// overwritten it, or a band's externals or steps do not fit.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace mcfd {

constexpr int kPipeChunk = 64;  // rows staged together

struct PipelineLimits {
  int ring, externals, steps;
};

struct PipelinePlanHost {
  int nc = 0, band_rows = 0, max_step = 0;
  bool ok = false;
  std::vector<int> chunk0;    // [nc + 1] first chunk of each band
  std::vector<int> rows;      // [nc] rows of each band
  std::vector<int> externals; // [nc]
  std::vector<int> step0;     // [nc + 1] first step of each band in steps (one closing entry per band)
  std::vector<int> steps;
  std::vector<int> pos, cell, count;     // [chunks * kPipeChunk]
  std::vector<unsigned short> slots;     // [..][4]
  std::vector<int> dest;                 // [..][4], -1: none
  std::vector<int> row_of_cell;          // [C] padded row index
};

inline bool plan_pipeline_host(const std::vector<int>& level_ptr, const std::vector<int>& pos_cell,
                               const std::vector<int>& ent_ptr, const std::vector<int>& ent_pos, int C, int nc,
                               int max_step, const PipelineLimits& lim, PipelinePlanHost& W) {
  W = PipelinePlanHost{};
  W.nc = nc;
  W.max_step = max_step;
  W.band_rows = std::max(1, (C + nc - 1) / nc);
  if (C <= 0 || C >= (1 << 24) * nc || lim.ring + lim.externals > (1 << 15)) return false;
  const int nlev = (int)level_ptr.size() - 1;
  std::vector<std::vector<int>> band(nc);  // positions
  std::vector<int> row_in_band(C), band_of(C), step_end(C);
  std::vector<std::vector<int>> step_first(nc);
  std::vector<std::vector<int>> step_most(nc);
  for (int l = 0; l < nlev; ++l) {
    std::vector<int> begin(nc);
    for (int k = 0; k < nc; ++k) begin[k] = (int)band[k].size();
    for (int p = level_ptr[l]; p < level_ptr[l + 1]; ++p) {
      const int k = pos_cell[p] / W.band_rows;
      band_of[p] = k;
      row_in_band[p] = (int)band[k].size();
      band[k].push_back(p);
    }
    for (int k = 0; k < nc; ++k)
      for (int f = begin[k]; f < (int)band[k].size(); f += max_step) {
        const int e = std::min(f + max_step, (int)band[k].size());
        int most = 0;
        for (int r = f; r < e; ++r) {
          const int p = band[k][r];
          most = std::max(most, ent_ptr[p + 1] - ent_ptr[p]);
          step_end[p] = e;
        }
        if (most > 4) return false;
        step_first[k].push_back(f);
        step_most[k].push_back(most);
      }
  }
  W.chunk0.assign(nc + 1, 0);
  W.rows.resize(nc);
  W.step0.assign(nc + 1, 0);
  for (int k = 0; k < nc; ++k) {
    const int n = (int)band[k].size();
    if ((int)step_first[k].size() > lim.steps) return false;
    W.rows[k] = n;
    W.chunk0[k + 1] = W.chunk0[k] + (n + kPipeChunk - 1) / kPipeChunk;
    for (size_t s = 0; s < step_first[k].size(); ++s) W.steps.push_back(step_first[k][s] | (step_most[k][s] << 24));
    W.steps.push_back(n);
    W.step0[k + 1] = (int)W.steps.size();
  }
  const size_t padded = (size_t)W.chunk0[nc] * kPipeChunk;
  W.pos.assign(padded, -1);
  W.cell.assign(padded, 0);
  W.count.assign(padded, 0);
  W.slots.assign(4 * padded, 0);
  W.dest.assign(4 * padded, -1);
  W.row_of_cell.assign(C, 0);
  W.externals.assign(nc, 0);
  std::vector<int> ext_slot(C, -1), ext_mark(C, -1);  // per position: slot and band of its last registration
  auto padded_row = [&](int p) { return (size_t)W.chunk0[band_of[p]] * kPipeChunk + row_in_band[p]; };
  for (int k = 0; k < nc; ++k) {
    int next = lim.ring;
    for (int r = 0; r < (int)band[k].size(); ++r) {
      const int p = band[k][r];
      const size_t i = padded_row(p);
      W.pos[i] = p;
      W.cell[i] = pos_cell[p];
      W.row_of_cell[pos_cell[p]] = (int)i;
      const int n = ent_ptr[p + 1] - ent_ptr[p];
      W.count[i] = n;
      for (int e = 0; e < n; ++e) {
        const int q = ent_pos[ent_ptr[p] + e];
        if (band_of[q] == k) {
          // the step's own rows may already have taken their ring slots
          if (row_in_band[q] < step_end[p] - lim.ring) return false;
          W.slots[4 * i + e] = (unsigned short)(row_in_band[q] & (lim.ring - 1));
          continue;
        }
        if (ext_mark[q] != k) {
          ext_mark[q] = k;
          ext_slot[q] = next++;
          if (next > lim.ring + lim.externals) return false;
          const size_t o = padded_row(q);
          int d = 0;
          while (d < 4 && W.dest[4 * o + d] >= 0) ++d;
          if (d == 4) return false;
          W.dest[4 * o + d] = (k << 16) | ext_slot[q];
        }
        W.slots[4 * i + e] = (unsigned short)(0x8000 | ext_slot[q]);
      }
    }
    W.externals[k] = next - lim.ring;
  }
  W.ok = true;
  return true;
}

// Cycles the plan's slowest band spends on its own steps, for choosing the
// rows per step: a step of one group of 16 rows is bound by the latency of its
// FP64 chain, of two groups by the SM's FP64 issue (measured in
// mcfd_pipeline.cu).
inline long long pipeline_cost(const PipelinePlanHost& W, int cycles_per_step) {
  int most = 0;
  for (int k = 0; k < W.nc; ++k) most = std::max(most, W.step0[k + 1] - W.step0[k]);
  return (long long)most * cycles_per_step;
}

}  // namespace mcfd
