// The pipelined band LU-SGS sweep: the forward and backward triangular solves
// of lusgs_apply on one thread-block cluster, with no barrier between blocks.
//
// Block k of the cluster owns a band of consecutive cells and solves their
// rows in sweep order (mcfd_pipeline_plan.h).  The bands depend on one
// another in one direction only, so the blocks run as a pipeline: a block
// pushes each solution another band reads into a slot of that block's shared
// memory (distributed shared memory, one 8-byte store per component), and the
// reader waits on the value itself, which starts as a NaN pattern that no
// arithmetic returns.  There is no flag, fence or barrier on the way, every
// slot is written once, and the hand-over's latency only delays the next
// band, not each level.
//
// What bounds a sweep is the dependent chain of a row, once per level: on
// GB300 an SM sub-partition's FP64 pipe takes one warp instruction per 64
// cycles, whatever the active lanes, and a row needs eight (two products, two
// differences, four for the quotient).  So:
// * the four components of a row are independent systems: a warp takes 16 rows
//   of two components and has a sub-partition to itself, and the two warps of
//   a step never wait for each other (steps of up to 32 rows: two such pairs,
//   a barrier of 64 threads between the two warps of one pair of components);
// * everything of a row that does not depend on the solutions is staged ahead
//   by bulk copies (one warp issues them, chunks of 64 rows laid out by field
//   so that no access has a bank conflict) and loaded while the previous
//   step's chain runs;
// * two more warps do the global stores and the pushes, behind the solvers;
// * the rows solved last stay in a ring in shared memory, so a step is: read
//   the entries' solutions, one product and difference per entry, the
//   quotient, store, synchronise the warp; no predicated FP64 instruction
//   (absent entries are products of zeros) and few others, since a warp alone
//   on its scheduler pays every instruction's latency.
// 512 x 256 bump (131,072 cells, 767 levels of at most 256 rows): 719 us per
// application (two sweeps, ~900 cycles a level) against 1,266 us of the
// windowed sweep, which bars the cluster once per window; 301 x 149 bump 433
// against 706, 3,050 triangles 119 against 144 us.
// The arithmetic is sweep_solve's in mcfd_implicit.cu, component by component:
// the same bits as every other schedule.  The forward sweep writes its
// solution times the clamped diagonal straight into the backward sweep's
// staged right-hand sides.
//
// Every wait is bounded by a number of polls, enough for the longest plan (a
// one-cell-wide strip, whose bands run one after another).  One that runs out
// sets MCFD_S_SWEEP_TIMEOUT and ends its warp's waiting: a solver goes on with
// whatever is there, a publisher stores and pushes nothing any more.  What a
// warp may then still touch is in bounds: the staged rows' slots start as
// zeros and are only ever replaced by the plan's, a chunk is copied only when
// the one before it in its place has landed, and the copying warp waits for
// the copies that it issued.  All blocks reach the closing cluster barrier,
// which keeps each block's shared memory alive until the last push arrived.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "mcfd_device.cuh"
#include "mcfd_implicit.h"
#include "mcfd_pipeline_plan.h"

namespace cg = cooperative_groups;

namespace mcfd {
namespace {

constexpr int kRing = 2048;       // own solutions kept: 64 KiB
constexpr int kExternals = 2046;  // slots for other bands' solutions: 64 KiB
constexpr int kZeroSlot = kRing + kExternals;  // always 0.0: the solution of an absent entry
constexpr int kSlots = kZeroSlot + 1;          // slot offsets (16 bytes each) fit 16 bits
static_assert(kSlots * 16 <= 1 << 16, "slot offsets");
constexpr int kMaxSteps = 6000;   // per band
constexpr int kStages = 4;        // chunks in flight (a power of two)
constexpr int kStagedRows = kStages * kPipeChunk;
// a chunk by field, 64 rows each, offsets in bytes: (diagonal, RN(1 /
// diagonal)), (first two values), (last two values), (four 16-bit slot
// offsets, output index, first destination), right-hand sides of the first
// and of the second pair of components, clamped diagonal; in shared memory
// every field is a ring of kStagedRows rows
constexpr int F_DIAG = 0, F_VAL01 = 1024, F_VAL23 = 2048, F_META = 3072, F_RHS = 4096, F_CLAMP = 6144;
constexpr int kChunkBytes = 6656, kChunkDoubles = kChunkBytes / 8;
constexpr unsigned kEmptyHi = 0x7ff4a5a5u;  // high word of a signalling NaN: no arithmetic result
// Polls a wait may take: one that may have to outlast the steps of all other
// bands in sequence, of the longest plan (a step takes up to 1,050 cycles and a
// poll at least 20, so 128 polls a step cover it more than twice; 16.5 M polls
// of some 100 cycles pass in a second), and one for a copy to land.
// Compile-time: as a launch argument the limit made the waiting loops 2 % of
// the small meshes' sweeps slower.
#ifndef MCFD_PIPELINE_SPINS
#define MCFD_PIPELINE_SPINS (16 * kMaxSteps * 128 + (1 << 22))
#endif
constexpr int kSpins = MCFD_PIPELINE_SPINS, kCopySpins = 1 << 22;
// a step's word: first row, rows - 1, then flags
constexpr unsigned W_MANY = 1u << 29;  // rows of more than two entries
constexpr unsigned W_WAIT = 1u << 30;  // its last row opens a chunk
constexpr unsigned W_FREE = 1u << 31;  // its first row leaves one

constexpr int kOffStage = (kSlots * 32 + 127) / 128 * 128;
constexpr int kOffSteps = kOffStage + kStages * kChunkBytes;
constexpr int kOffBars = kOffSteps + ((kMaxSteps + 8) * 4 + 15) / 16 * 16;
constexpr int kOffProgress = kOffBars + 2 * kStages * 8;
constexpr int kSmemBytes = kOffProgress + 16;
static_assert(kSmemBytes <= 227 * 1024, "the pipelined sweep's shared memory");

struct PipeDev {
  const double* stage;
  const int *chunk0, *rows, *externals, *step0;
  const unsigned* steps;
  const int4* dest;  // every row's destinations
  double* out;       // backward: [C][4]; forward: the backward plan's stage
  DevStatus* status;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int spins) {
  for (int i = 0; i < spins; ++i)
    if (mbar_try(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ unsigned remote(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void push(unsigned addr, double v) {
  asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(addr), "l"(__double_as_longlong(v)) : "memory");
}
__device__ __forceinline__ double poll(unsigned addr) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void st_shared(unsigned addr, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ bool empty(double x) { return (unsigned)(ia::bits(x) >> 32) == kEmptyHi; }

// What div_rn_fma leaves to the exact division, out of the step's way: a zero
// dividend (q0 = a y is the signed zero), the ends of the range, candidates
// next to a rounding boundary.
__device__ __noinline__ double quotient_slow(double a, double b, double q0) {
  return (ia::bits(a) << 1) == 0ull && (ia::bits(q0) << 1) == 0ull ? q0 : div_rn(a, b);
}

// a / b as div_rn_fma computes it (the same candidate and remainder test)
// with fewer instructions around its four FP64 operations: the warp runs
// alone on its scheduler, so each one delays the next level.  y = RN(1/b), or
// NaN where b's exponent is outside 2^+-200 (k_pipeline_values), so the
// quotient's exponent alone decides the range; a quotient whose significand
// is zero (a power of two, whose neighbours differ by side) goes to the slow
// path, and so does a remainder that only the low words would accept.  hb:
// high word of |b|, less 1076 in the exponent field.
__device__ __forceinline__ double quotient(double a, double b, double y, unsigned hb) {
  const double q0 = __dmul_rn(a, y);
  const double q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
  const double r = __fma_rn(-b, q, a);
  const unsigned long long iq = ia::bits(q);
  const unsigned qh = (unsigned)(iq >> 32), rh = (unsigned)(ia::bits(r) >> 32) & 0x7fffffffu;
  const unsigned qe = qh & 0x7ff00000u;
  // |r| < |b| u / 2 with u the spacing of doubles at q: |b| 2^(eq - 1076)
  if (qe - (300u << 20) < (1400u << 20) && ((qh & 0xfffffu) | (unsigned)iq) != 0u && rh < hb + qe) return q;
  return quotient_slow(a, b, q0);
}

// The third and fourth entry's terms, behind a call: inlined, the compiler
// predicates them, and four predicated-off FP64 instructions cost a step of
// two-entry rows 256 cycles.
__device__ __noinline__ double more_terms(double acc, double v2, double x2, double v3, double x3) {
  acc = acc - v2 * x2;
  return acc - v3 * x3;
}

// Everything of a row that does not depend on the solutions.
struct PipeRow {
  double diag, inv, rhs, v0, v1;
  unsigned s01, at;   // entries' slot offsets, offset of the row's staged fields
  unsigned to, word;  // address of its own solution; the step's word
};

// GROUPS: warps per pair of components, 16 rows of a step each.  Warps 0 ..
// 2 GROUPS - 1 solve, the next two publish (global stores and pushes, one for
// each pair of components), the last one copies.
template <int GROUPS, bool FORWARD>
__global__ void __launch_bounds__(32 * (2 * GROUPS + 3), 1) k_lusgs_pipeline(PipeDev a) {
  extern __shared__ __align__(128) unsigned char smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int band = (int)cluster.block_rank();
  double* sl = reinterpret_cast<double*>(smem);  // [2 component pairs][kSlots][2]
  unsigned* steps = reinterpret_cast<unsigned*>(smem + kOffSteps);
  const unsigned bars = smem_u32(smem + kOffBars);  // full[kStages], free[kStages]
  const unsigned char* staged = smem + kOffStage;
  const unsigned stage = smem_u32(staged), progress = smem_u32(smem + kOffProgress);
  const int nt = (int)blockDim.x, t = (int)threadIdx.x, warp = t >> 5, lane = t & 31;
  const int n_steps = a.step0[band + 1] - a.step0[band];
  const int n_chunks = (a.rows[band] + kPipeChunk - 1) / kPipeChunk;
  if (t == 0)
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bars + 8 * i, 1);
      mbar_init(bars + 8 * (kStages + i), 2 * GROUPS + 2);
    }
  if (t < 4) reinterpret_cast<int*>(smem + kOffProgress)[t] = 0;
  for (int i = t; i < 4 * a.externals[band]; i += nt) {  // both pairs' [externals][2]
    const int pair = i & 1, e = i >> 1;
    reinterpret_cast<unsigned long long*>(sl)[(size_t)pair * kSlots * 2 + 2 * kRing + e] = (unsigned long long)kEmptyHi << 32;
  }
  if (t < 4) sl[(size_t)(t & 1) * kSlots * 2 + 2 * kZeroSlot + (t >> 1)] = 0.0;
  if (warp == 2 * GROUPS + 2)
    for (int i = lane; i < kStagedRows; i += 32)
      reinterpret_cast<uint4*>(smem + kOffStage + kStages * F_META)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = t; i < n_steps; i += nt) steps[i] = a.steps[a.step0[band] + i];
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  cluster.sync();  // every block's slots are empty before the first push
  bool dead = false;  // a bounded wait ran out: no further waiting
  // a consumer of the staged chunks: how many it knows to have landed and has
  // handed back (every row before the step's first is done with)
  int ready = 0, freed = 0;
  auto chunks_of = [&](unsigned w) {
    if (w & W_WAIT) {
      if (!dead) dead = !mbar_wait(bars + 8 * (ready % kStages), (ready / kStages) & 1, kSpins);
      ++ready;
    }
    if (w & W_FREE) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (kStages + freed % kStages));
      ++freed;
    }
  };
  if (warp == 2 * GROUPS + 2) {
    // ---- the copies, kStages chunks ahead, one per field of a chunk
    if (lane == 0) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(a.stage) + (size_t)a.chunk0[band] * kChunkBytes;
      int issued = 0;
      for (; issued < n_chunks; ++issued, src += kChunkBytes) {
        const int s = issued % kStages, use = issued / kStages;
        if (use > 0)  // handed back, and landed (a warp that stopped waiting hands back early)
          dead = !mbar_wait(bars + 8 * (kStages + s), (use - 1) & 1, kSpins) ||
                 !mbar_wait(bars + 8 * s, (use - 1) & 1, kCopySpins);
        if (dead) break;  // the solvers' own waits run out too
        mbar_expect(bars + 8 * s, kChunkBytes);
#pragma unroll
        for (int f = 0; f < 6; ++f)
          bulk_load(stage + kStages * 1024 * f + 1024 * s, src + 1024 * f, 1024, bars + 8 * s);
        bulk_load(stage + kStages * F_CLAMP + 512 * s, src + F_CLAMP, 512, bars + 8 * s);
      }
      // no copy may be in flight when the block ends
      for (int c = issued > kStages ? issued - kStages : 0; c < issued; ++c)
        if (!mbar_wait(bars + 8 * (c % kStages), (c / kStages) & 1, kCopySpins)) dead = true;
    }
  } else if (warp >= 2 * GROUPS) {
    // ---- publishing: the solved rows of each step, behind the solvers
    const int pair = warp & 1, half = lane >> 4, comp = 2 * pair + half;
    const unsigned mine = smem_u32(sl + (size_t)pair * kSlots * 2 + half);
    for (int s = 0; s < n_steps; ++s) {
      const unsigned w = steps[s];
      chunks_of(w);
      for (int g = 0; g < GROUPS; ++g) {
        int spins = 0;
        while (!dead) {
          int done;
          asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(done) : "r"(progress + 4u * (2 * g + pair)) : "memory");
          if (done > s) break;
          if (++spins > kSpins) dead = true;
        }
      }
      dead = __any_sync(0xffffffffu, dead);
      if (dead) break;
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        const int k = 16 * g + (lane & 15);
        if (k > (int)(w >> 24 & 31u)) continue;
        const int row = (int)(w & 0xffffffu) + k;
        const unsigned r = (unsigned)row & (kStagedRows - 1);
        const int4 meta = reinterpret_cast<const int4*>(staged + kStages * F_META)[r];
        const unsigned out = (unsigned)meta.z;
        const int dest = meta.w;
        const double res = sl[(size_t)pair * kSlots * 2 + 2 * ((unsigned)row & (kRing - 1)) + half];
        if (dest >= 0) {
          push(remote(mine + 16u * ((unsigned)dest & 0xffffu), ((unsigned)dest & 0x3fffffffu) >> 16), res);
          if (dest & 0x40000000) {
            const int4 m = a.dest[(size_t)a.chunk0[band] * kPipeChunk + row];
            const int more[3] = {m.y, m.z, m.w};
#pragma unroll
            for (int i = 0; i < 3; ++i)
              if (more[i] >= 0) push(remote(mine + 16u * (unsigned)(more[i] & 0xffff), (unsigned)(more[i] >> 16)), res);
          }
        }
        // forward: out is the first component's right-hand side in the
        // backward stage, a pair of components [row][2], pairs 128 doubles apart
        if (FORWARD) a.out[(size_t)out + 128 * pair + half] = reinterpret_cast<const double*>(staged + kStages * F_CLAMP)[r] * res;
        else a.out[4 * (size_t)out + comp] = res;
      }
      __syncwarp();
    }
  } else if (n_steps > 0) {
    // ---- solving: warp = (group, pair), lane = (component of the pair, row).
    // Lanes beyond a step's rows repeat its last row: the same values to the
    // same places, and no predicates.
    const int pair = warp & 1, group = warp >> 1, half = lane >> 4;
    const unsigned r16 = 16 * group + (lane & 15);
    const unsigned mine = smem_u32(sl + (size_t)pair * kSlots * 2 + half);
    const double* rhs = reinterpret_cast<const double*>(staged + kStages * (F_RHS + 1024 * pair)) + half;
    auto load = [&](unsigned w, PipeRow& R) {
      const unsigned row = (w & 0xffffffu) + min(r16, w >> 24 & 31u);
      const unsigned i = row & (kStagedRows - 1);
      const double2 d = reinterpret_cast<const double2*>(staged + kStages * F_DIAG)[i];
      const double2 v01 = reinterpret_cast<const double2*>(staged + kStages * F_VAL01)[i];
      R.s01 = reinterpret_cast<const uint4*>(staged + kStages * F_META)[i].x;
      R.rhs = rhs[2 * i];
      R.diag = d.x;
      R.inv = d.y;
      R.v0 = v01.x;
      R.v1 = v01.y;
      R.at = 16u * i;
      R.to = mine + 16u * (row & (kRing - 1));
      R.word = w;
    };
    auto announce = [&](int done) {  // steps solved, to the publishing warp
      if (lane == 0)
        asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(progress + 4u * warp), "r"(done) : "memory");
    };
    unsigned after = n_steps > 1 ? steps[1] : 0u;  // the next step's word
    auto step = [&](int s, const PipeRow& R, PipeRow& N) {
      const unsigned w = after;
      after = s + 2 < n_steps ? steps[s + 2] : 0u;
      const unsigned a0 = mine + (R.s01 & 0xffffu), a1 = mine + (R.s01 >> 16);
      double x0 = poll(a0), x1 = poll(a1), x2 = 0.0, x3 = 0.0, v2 = 0.0, v3 = 0.0;
      unsigned a2 = 0, a3 = 0;
      if (R.word & W_MANY) {
        const unsigned s23 = *reinterpret_cast<const unsigned*>(staged + kStages * F_META + R.at + 4);
        const double2 v23 = *reinterpret_cast<const double2*>(staged + kStages * F_VAL23 + R.at);
        a2 = mine + (s23 & 0xffffu);
        a3 = mine + (s23 >> 16);
        v2 = v23.x;
        v3 = v23.y;
        x2 = poll(a2);
        x3 = poll(a3);
      }
      if (__any_sync(0xffffffffu, empty(x0) | empty(x1) | empty(x2) | empty(x3))) {
        // another band's row has not arrived yet; what it waits for may be
        // this warp's own last step, so that is announced first
        announce(s);
        for (int spins = 0; __any_sync(0xffffffffu, empty(x0) | empty(x1) | empty(x2) | empty(x3)); ++spins) {
          if (__any_sync(0xffffffffu, dead) || spins > kSpins) {  // the lanes leave together
            dead = true;
            break;
          }
          x0 = poll(a0);
          x1 = poll(a1);
          if (R.word & W_MANY) {
            x2 = poll(a2);
            x3 = poll(a3);
          }
        }
      }
      const double p0 = R.v0 * x0, p1 = R.v1 * x1;
      announce(s);
      if (w & (W_WAIT | W_FREE)) chunks_of(w);  // this step's staged fields have all been read
      load(w, N);  // the next step's rows while this step's chain runs (after the last: unused)
      double acc = R.rhs - p0;
      acc = acc - p1;
      if (R.word & W_MANY) acc = more_terms(acc, v2, x2, v3, x3);
      const unsigned hb = ((unsigned)(ia::bits(R.diag) >> 32) & 0x7fffffffu) - (1076u << 20);
      st_shared(R.to, quotient(acc, R.diag, R.inv, hb));
      __syncwarp();
      if (GROUPS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + pair), "r"(32 * GROUPS) : "memory");
    };
    PipeRow A, B;
    chunks_of(steps[0]);
    load(steps[0], A);
    for (int s = 0; s < n_steps; s += 2) {
      step(s, A, B);
      if (s + 1 < n_steps) step(s + 1, B, A);
    }
    announce(n_steps);
  }
  if (dead) atomicOr(&a.status->code, MCFD_S_SWEEP_TIMEOUT);
  __syncwarp();
  cluster.sync();
}

// Values of the staged rows after an assembly (pk_row: diagonal, RN(1 /
// diagonal), fixed-point reciprocal, clamped diagonal, four values; absent
// entries have the value 0.0 and read the slot that holds 0.0, so their
// difference changes no bit).
__global__ void k_pipeline_values(int n, const int* __restrict__ pos, const double2* __restrict__ pk_row,
                                  unsigned char* __restrict__ stage) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = pos[i];
  if (p < 0) return;
  const double2 q0 = pk_row[4 * (size_t)p], q1 = pk_row[4 * (size_t)p + 1], q2 = pk_row[4 * (size_t)p + 2],
                q3 = pk_row[4 * (size_t)p + 3];
  unsigned char* b = stage + (size_t)(i / kPipeChunk) * kChunkBytes;
  const int r = i % kPipeChunk;
  // the quotient's shortcut takes divisors within 2^+-200 (quotient)
  const int e = (int)(ia::bits(q0.x) >> 52) & 0x7ff;
  const double inv = e >= 823 && e <= 1223 ? q0.y : __longlong_as_double(0x7ff8000000000000ll);
  reinterpret_cast<double2*>(b + F_DIAG)[r] = make_double2(q0.x, inv);
  reinterpret_cast<double2*>(b + F_VAL01)[r] = q2;
  reinterpret_cast<double2*>(b + F_VAL23)[r] = q3;
  reinterpret_cast<double*>(b + F_CLAMP)[r] = q1.y;
}

// Right-hand sides of a forward sweep.
__global__ void k_pipeline_rhs(int n, const int* __restrict__ cell, const int* __restrict__ pos,
                               const double* __restrict__ in, unsigned char* __restrict__ stage) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || pos[i] < 0) return;
  const St4 v = ld4(in + 4 * (size_t)cell[i]);
  double2* b = reinterpret_cast<double2*>(stage + (size_t)(i / kPipeChunk) * kChunkBytes + F_RHS) + i % kPipeChunk;
  b[0] = make_double2(v.a, v.b);
  b[kPipeChunk] = make_double2(v.c, v.d);
}

template <int GROUPS, bool FORWARD>
bool cluster_fits(int nc) {
  auto kernel = k_lusgs_pipeline<GROUPS, FORWARD>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) return false;
  if (nc > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return false;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(32 * (2 * GROUPS + 3));
  cfg.dynamicSmemBytes = kSmemBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  return cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
}

template <int GROUPS, bool FORWARD>
cudaError_t launch(const SweepPipeline& p, double* out, DevStatus* status, cudaStream_t s) {
  const PipeDev a{p.stage, p.chunk0, p.rows, p.externals, p.step0, reinterpret_cast<const unsigned*>(p.steps),
                  reinterpret_cast<const int4*>(p.dest), out, status};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.nc);
  cfg.blockDim = dim3(32 * (2 * GROUPS + 3));
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, k_lusgs_pipeline<GROUPS, FORWARD>, a);
}

inline int blocks_for(int n) { return (n + 255) / 256; }

}  // namespace

bool pipeline_available(int nc) {
  const bool ok = cluster_fits<1, true>(nc) && cluster_fits<1, false>(nc) && cluster_fits<2, true>(nc) &&
                  cluster_fits<2, false>(nc);
  cudaGetLastError();  // clear a refused attribute's error
  return ok;
}

void pipeline_free(SweepPipeline& p) {
  for (void* q : p.owned) cudaFree(q);
  p = SweepPipeline{};
}

// Cycles per step: measured ~930 for one group; two groups add a barrier of 64
// threads and the contention of four solving warps with the other three.
constexpr int kCycles1 = 930, kCycles2 = 1050;

cudaError_t pipeline_plan(SweepPlan& fwd, SweepPlan& bwd, int C, int nc) {
  pipeline_free(fwd.pipe);
  pipeline_free(bwd.pipe);
  PipelinePlanHost H[2];
  SweepPlan* pl[2] = {&fwd, &bwd};
  const PipelineLimits lim{kRing, kExternals, kMaxSteps};
  for (int d = 0; d < 2; ++d) {
    // one launch sweeps every level: levels of the grid launches are not planned
    for (const SweepPlan::Launch& l : pl[d]->schedule)
      if (!l.wavefront || l.l0 != 0 || l.l1 != pl[d]->n_levels) return cudaSuccess;
    PipelinePlanHost two;
    const bool one = plan_pipeline_host(pl[d]->host_level_ptr, pl[d]->host_pos_cell, pl[d]->host_ent_ptr,
                                        pl[d]->host_ent_pos, C, nc, 16, lim, H[d]);
    if (!plan_pipeline_host(pl[d]->host_level_ptr, pl[d]->host_pos_cell, pl[d]->host_ent_ptr, pl[d]->host_ent_pos, C,
                            nc, 32, lim, two)) {
      if (!one) return cudaSuccess;
    } else if (!one || pipeline_cost(two, kCycles2) < pipeline_cost(H[d], kCycles1)) {
      H[d] = std::move(two);
    }
  }
  for (int d = 0; d < 2; ++d) {
    SweepPipeline& p = pl[d]->pipe;
    const PipelinePlanHost& h = H[d];
    const size_t padded = h.pos.size(), chunks = padded / kPipeChunk;
    if (chunks * kChunkDoubles > (size_t)1 << 31) return cudaSuccess;
    p.nc = nc;
    p.groups = h.max_step / 16;
    p.n_padded = (int)padded;
    // the topology fields of the stage; values and right-hand sides follow
    std::vector<double> st(chunks * kChunkDoubles, 0.0);
    for (size_t i = 0; i < padded; ++i) {
      if (h.pos[i] < 0) continue;
      unsigned char* b = reinterpret_cast<unsigned char*>(st.data()) + i / kPipeChunk * kChunkBytes;
      unsigned short slot[4];
      for (int k = 0; k < 4; ++k)
        slot[k] = (unsigned short)(16 * (k < h.count[i] ? h.slots[4 * i + k] & 0x7fff : kZeroSlot));
      int m[4] = {0, 0, h.cell[i], h.dest[4 * i]};
      memcpy(m, slot, 8);
      if (d == 0) {  // forward: the cell's first right-hand side in the backward stage
        const size_t j = (size_t)H[1].row_of_cell[h.cell[i]];
        m[2] = (int)(j / kPipeChunk * kChunkDoubles + F_RHS / 8 + 2 * (j % kPipeChunk));
      }
      if (h.dest[4 * i + 1] >= 0) m[3] |= 0x40000000;
      memcpy(b + F_META + 16 * (i % kPipeChunk), m, 16);
    }
    // the steps' words (no closing entries)
    std::vector<int> words, step0(nc + 1, 0);
    for (int k = 0; k < nc; ++k) {
      int chunk_last = -1, chunk_first = 0;
      for (int q = h.step0[k]; q + 1 < h.step0[k + 1]; ++q) {
        const int f = h.steps[q] & 0xffffff, e = h.steps[q + 1] & 0xffffff;
        unsigned w = (unsigned)f | (unsigned)(e - f - 1) << 24;
        if (h.steps[q] >> 24 > 2) w |= W_MANY;
        if ((e - 1) / kPipeChunk > chunk_last) w |= W_WAIT, ++chunk_last;
        if (f / kPipeChunk > chunk_first) w |= W_FREE, ++chunk_first;
        words.push_back((int)w);
      }
      step0[k + 1] = (int)words.size();
    }
    cudaError_t e = cudaSuccess;
    auto put = [&](const void* src, size_t bytes, void** dst) {
      if (e != cudaSuccess) return;
      e = cudaMalloc(dst, std::max<size_t>(bytes, 16));
      if (e != cudaSuccess) return;
      p.owned.push_back(*dst);
      if (bytes) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
    };
    auto ints = [&](const std::vector<int>& v, int** dst) { put(v.data(), v.size() * sizeof(int), (void**)dst); };
    put(st.data(), st.size() * sizeof(double), (void**)&p.stage);
    ints(h.chunk0, &p.chunk0);
    ints(h.rows, &p.rows);
    ints(h.externals, &p.externals);
    ints(step0, &p.step0);
    ints(words, &p.steps);
    ints(h.pos, &p.pos);
    ints(h.cell, &p.cell);
    ints(h.dest, &p.dest);
    if (e != cudaSuccess) return e;
  }
  fwd.pipe.ok = bwd.pipe.ok = true;
  return cudaSuccess;
}

cudaError_t pipeline_values(SweepPlan& pl, cudaStream_t s) {
  if (!pl.pipe.ok || pl.pipe.n_padded == 0) return cudaSuccess;
  count_launch();
  k_pipeline_values<<<blocks_for(pl.pipe.n_padded), 256, 0, s>>>(pl.pipe.n_padded, pl.pipe.pos, pl.pk_row,
                                                                  reinterpret_cast<unsigned char*>(pl.pipe.stage));
  return cudaGetLastError();
}

cudaError_t pipeline_apply(SweepPlan& fwd, SweepPlan& bwd, const double* v, double* x, DevStatus* status,
                           cudaStream_t s) {
  count_launch();
  k_pipeline_rhs<<<blocks_for(fwd.pipe.n_padded), 256, 0, s>>>(fwd.pipe.n_padded, fwd.pipe.cell, fwd.pipe.pos, v,
                                                               reinterpret_cast<unsigned char*>(fwd.pipe.stage));
  cudaError_t e = fwd.pipe.groups == 1 ? launch<1, true>(fwd.pipe, bwd.pipe.stage, status, s)
                                       : launch<2, true>(fwd.pipe, bwd.pipe.stage, status, s);
  if (e == cudaSuccess)
    e = bwd.pipe.groups == 1 ? launch<1, false>(bwd.pipe, x, status, s) : launch<2, false>(bwd.pipe, x, status, s);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace mcfd
