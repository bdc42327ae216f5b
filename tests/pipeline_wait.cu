// The pipelined sweep (meshcfd_gb300/csrc/mcfd_pipeline.cu, compiled into this
// program) where its waits are longest: a one-cell-wide strip of the most steps
// a plan may have, whose bands run one after another, and a grid of two groups
// of rows a step, each against the substitution on the host bit for bit.
// Compiled with -DMCFD_PIPELINE_SPINS=<polls>, where its waits run out: the
// kernels must end, report MCFD_S_SWEEP_TIMEOUT (or be right) and leave the
// plan's staged rows as they were, right-hand sides aside.
//
// usage: pipeline_wait -> "cases=<n> timeouts=<n> failures=<n>", 77 without a cluster
#ifdef MCFD_PIPELINE_SPINS
static const int polls = MCFD_PIPELINE_SPINS;
#else
static const int polls = -1;
#endif

#include <cstdio>
#include <cstdlib>

#include "../meshcfd_gb300/csrc/mcfd_pipeline.cu"

namespace mcfd {
void count_launch(int) {}
}  // namespace mcfd

using namespace mcfd;

#define CUDA(call)                                                                  \
  do {                                                                              \
    const cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                        \
      std::printf("%s: %s\n", #call, cudaGetErrorString(e_));                       \
      std::exit(1);                                                                 \
    }                                                                               \
  } while (0)

static unsigned long long g_state = 7;
static double uniform() {
  unsigned long long z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
}

// One sweep over nx x ny cells (neighbours c +- 1 in a mesh row, c +- nx),
// rows by (level, cell), lower or higher neighbours with the weight of a pair.
struct Rows {
  SweepPlan plan;
  std::vector<double> val;  // per entry
  std::vector<double2> pk;  // pk_row
};

static double weight(int a, int b) {
  unsigned long long z = ((unsigned long long)(a < b ? a : b) << 32 | (unsigned)(a < b ? b : a)) * 0x9e3779b97f4a7c15ull;
  z ^= z >> 29;
  return (double)(z >> 12) * 0x1p-53 - 0.25;
}

static void make(Rows& S, int nx, int ny, bool forward, const std::vector<double>& diag, const std::vector<double>& clamp) {
  const int C = nx * ny;
  auto entries = [&](int c, int out[2]) {
    int n = 0;
    const int i = c % nx, j = c / nx;
    if (forward) {
      if (j > 0) out[n++] = c - nx;
      if (i > 0) out[n++] = c - 1;
    } else {
      if (i + 1 < nx) out[n++] = c + 1;
      if (j + 1 < ny) out[n++] = c + nx;
    }
    return n;
  };
  SweepPlan& p = S.plan;
  p.n_levels = nx + ny - 1;
  std::vector<int> level(C), pos(C);
  p.host_level_ptr.assign(p.n_levels + 1, 0);
  for (int c = 0; c < C; ++c) {
    const int l = c % nx + c / nx;
    level[c] = forward ? l : p.n_levels - 1 - l;
    p.host_level_ptr[level[c] + 1]++;
  }
  for (int l = 0; l < p.n_levels; ++l) p.host_level_ptr[l + 1] += p.host_level_ptr[l];
  std::vector<int> fill(p.host_level_ptr.begin(), p.host_level_ptr.end() - 1);
  p.host_pos_cell.resize(C);
  for (int c = 0; c < C; ++c) {
    pos[c] = fill[level[c]]++;
    p.host_pos_cell[pos[c]] = c;
  }
  p.host_ent_ptr.assign(1, 0);
  for (int q = 0; q < C; ++q) {
    int e[2];
    const int c = p.host_pos_cell[q], n = entries(c, e);
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k = 0; k < n; ++k) {
      p.host_ent_pos.push_back(pos[e[k]]);
      S.val.push_back(v[k] = weight(c, e[k]));
    }
    p.host_ent_ptr.push_back((int)p.host_ent_pos.size());
    S.pk.push_back(make_double2(diag[c], 1.0 / diag[c]));
    S.pk.push_back(make_double2(0.0, clamp[c]));
    S.pk.push_back(make_double2(v[0], v[1]));
    S.pk.push_back(make_double2(v[2], v[3]));
  }
  p.schedule.push_back({1, 0, p.n_levels});
  CUDA(cudaMalloc((void**)&p.pk_row, S.pk.size() * sizeof(double2)));
  CUDA(cudaMemcpy(p.pk_row, S.pk.data(), S.pk.size() * sizeof(double2), cudaMemcpyHostToDevice));
}

// (D + T) out = rhs, one component a column
static void solve(const Rows& S, const std::vector<double>& rhs, const std::vector<double>& diag, std::vector<double>& out) {
  const SweepPlan& p = S.plan;
  for (size_t q = 0; q < p.host_pos_cell.size(); ++q) {
    const int c = p.host_pos_cell[q];
    for (int k = 0; k < 4; ++k) {
      double acc = rhs[4 * c + k];
      for (int e = p.host_ent_ptr[q]; e < p.host_ent_ptr[q + 1]; ++e) {
        const double t = S.val[e] * out[4 * p.host_pos_cell[p.host_ent_pos[e]] + k];
        acc = acc - t;
      }
      out[4 * c + k] = acc / diag[c];
    }
  }
}

int main() {
  const int nc = pipeline_available(16) ? 16 : pipeline_available(8) ? 8 : 0;
  if (nc == 0) return 77;
  int cases = 0, timeouts = 0, failures = 0;
  const int sizes[][2] = {{nc * kMaxSteps, 1}, {1, nc * kMaxSteps}, {420, 260}, {50, 3}};
  for (const auto& size : sizes) {
    const int nx = size[0], ny = size[1], C = nx * ny;
    std::vector<double> diag(C), clamp(C), v(4 * (size_t)C), y(4 * (size_t)C), x(4 * (size_t)C);
    for (int c = 0; c < C; ++c) {
      diag[c] = 1.0 + uniform();
      clamp[c] = diag[c];
      for (int k = 0; k < 4; ++k) v[4 * c + k] = 2.0 * uniform() - 1.0;
    }
    Rows fwd, bwd;
    make(fwd, nx, ny, true, diag, clamp);
    make(bwd, nx, ny, false, diag, clamp);
    CUDA(pipeline_plan(fwd.plan, bwd.plan, C, nc));
    if (!fwd.plan.pipe.ok || !bwd.plan.pipe.ok) {
      std::printf("%d x %d: not planned\n", nx, ny);
      return 1;
    }
    solve(fwd, v, diag, y);
    for (size_t i = 0; i < y.size(); ++i) y[i] = clamp[i / 4] * y[i];
    solve(bwd, y, diag, x);
    double *dv, *dx;
    DevStatus* status;
    CUDA(cudaMalloc((void**)&dv, v.size() * sizeof(double)));
    CUDA(cudaMalloc((void**)&dx, v.size() * sizeof(double)));
    CUDA(cudaMalloc((void**)&status, sizeof(DevStatus)));
    CUDA(cudaMemcpy(dv, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice));
    CUDA(pipeline_values(fwd.plan, nullptr));
    CUDA(pipeline_values(bwd.plan, nullptr));
    auto staged = [&](const SweepPipeline& p) {
      std::vector<unsigned char> h((size_t)p.n_padded / kPipeChunk * kChunkBytes);
      CUDA(cudaMemcpy(h.data(), p.stage, h.size(), cudaMemcpyDeviceToHost));
      for (size_t o = 0; o < h.size(); o += kChunkBytes) std::memset(h.data() + o + F_RHS, 0, F_CLAMP - F_RHS);
      return h;
    };
    const auto plan_f = staged(fwd.plan.pipe), plan_b = staged(bwd.plan.pipe);
    std::vector<double> got(v.size());
    for (int repeat = 0; repeat < 3; ++repeat) {
      CUDA(cudaMemset(status, 0, sizeof(DevStatus)));
      CUDA(cudaMemset(dx, 0, v.size() * sizeof(double)));
      CUDA(pipeline_apply(fwd.plan, bwd.plan, dv, dx, status, nullptr));
      CUDA(cudaDeviceSynchronize());
      DevStatus st;
      CUDA(cudaMemcpy(&st, status, sizeof(st), cudaMemcpyDeviceToHost));
      CUDA(cudaMemcpy(got.data(), dx, got.size() * sizeof(double), cudaMemcpyDeviceToHost));
      const bool same = std::memcmp(got.data(), x.data(), x.size() * sizeof(double)) == 0;
      const bool kept = staged(fwd.plan.pipe) == plan_f && staged(bwd.plan.pipe) == plan_b;
      ++cases;
      if (st.code == MCFD_S_SWEEP_TIMEOUT) ++timeouts;
      const bool ok = kept && (st.code == 0 ? same && polls != 0 : st.code == MCFD_S_SWEEP_TIMEOUT && polls >= 0);
      if (!ok)
        ++failures, std::printf("%d x %d, %d polls: status %#x, %s, plan %s\n", nx, ny, polls, st.code,
                                same ? "same" : "different", kept ? "kept" : "changed");
    }
    pipeline_free(fwd.plan.pipe);
    pipeline_free(bwd.plan.pipe);
    cudaFree(fwd.plan.pk_row);
    cudaFree(bwd.plan.pk_row);
    cudaFree(dv);
    cudaFree(dx);
    cudaFree(status);
  }
  std::printf("cases=%d timeouts=%d failures=%d\n", cases, timeouts, failures);
  return failures ? 1 : 0;
}
