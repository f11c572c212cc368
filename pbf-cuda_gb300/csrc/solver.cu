// solver.cu — the per-particle passes of one step, in cell order:
//   reorder   gather pos/vel/iid by the sorted permutation, recompute x*
//   lambda    density rho_i and lambda_i        computeLambda  (fluids/Simulator_kernel.cuh:52-129)
//   delta_p   s_corr, clamp, wall clamp         computetpos    (fluids/Simulator_kernel.cuh:131-194)
//             the last iteration also writes v = (x_final - x) / dt and the
//             caller's permuted pos / iid       h_updateVelocity (fluids/Simulator.cu:127-137)
//   xsph      XSPH viscosity                    computeXSPH    (fluids/Simulator_kernel.cuh:196-239)
//
// Every pass is gather-only (no atomics on results, no cross-thread writes),
// so results are deterministic.  Neighbour semantics follow the reference
// exactly: the grid is built once per step from x*, every pass looks up the
// 3x3x3 cells around cell(current x_i) in that (stale) grid.  For each
// (dx, dy) column the three z-consecutive cells are adjacent in cell order,
// so the window is 9 runs of sorted slots, visited in the reference's order
// (dx outer, dy inner, slots ascending; fluids/Simulator_kernel.cuh:78-88).
// Jacobi iterations ping-pong between two position buffers instead of the
// reference's tpos -> npos copy (fluids/Simulator.cu:247-248).
//
// Each pass is two kernels.  The sparse kernel walks a particle's window in
// one thread (fluid at rest: ~200 candidates; a window whose grouped cells --
// see pbf_internal.cuh -- bring it under dense_window entries is walked group
// by group): the lambda pass lists the particle's hits, the delta_p passes of
// the iteration read the list.  In current-cell order a thread of the lambda
// and xsph passes takes two particles of one cell.  A particle whose
// window still exceeds dense_window entries (particles piled into a few
// cells) instead appends itself to a dense list; the persistent dense kernel
// takes the list in batches of 32 particles from a counter, splits each
// batch's windows over dense_split warps (each walking one part of every
// lane's window) and adds the parts' partial sums in part order in shared
// memory.  Steps of fewer than kDenseAllBelow particles send every particle
// to the dense kernel by default (one thread per particle would leave most
// SMs idle).  Both orders are fixed, so results stay deterministic; they
// differ from the reference's sequential sums only by rounding.  The walks
// test chunks of 32 candidates into hit masks and run the pair body on the
// hits, through a queue of masks (the dense kernel: optionally); the dense
// kernel has a variant that stages its block's column runs in shared memory
// by bulk asynchronous copies.  None of this changes any sum.
//
// Particles piled onto one position (a grouped cell's position group) have
// bitwise the same window, position and, within a step, lambda: their lambda
// and delta_p results are equal.  When a step has grouped cells, each lambda
// pass first builds a work list (k_work_mark, k_work_list: one particle per
// position group plus every particle outside the groups, in cell order), the
// two passes run on that list, and k_follow copies each group's results to
// its other members.  With no grouped cell the list is the identity and those
// kernels return at once.
//
// IEEE semantics follow the reference's: its kernels evaluate every
// candidate of the window, so a NaN distance (from a NaN position) poisons
// the sums, a non-finite lambda_j poisons delta_p through a zero gradient,
// and 0 * v / (rho_i + rho_j) is NaN when both densities are zero.  Here the
// candidate test is written NaN-inclusively (!(r2 >= h2), as the reference's
// `if (r2 >= h2) return 0`), and the two poisoning rules that need every
// candidate's lambda / density / velocity run only when a per-step flag says
// such a value exists (StepFlag); otherwise candidates outside the cutoff
// contribute exactly zero and are skipped.
#include <climits>

#include "pbf_internal.cuh"

namespace pbf {

namespace {

constexpr int kSparseThreads = 128;
// PBF_DENSE_WARPS (a build-time tuning macro): warps of a dense-kernel block,
// i.e. the chunks each listed particle's window is split into.
#ifndef PBF_DENSE_WARPS
#define PBF_DENSE_WARPS 8
#endif
constexpr int kDenseWarps = PBF_DENSE_WARPS;   // chunks of a dense item's windows
constexpr int kDenseThreads = 32 * kDenseWarps;
// Below kDenseAllBelow particles one thread per particle leaves most of the
// GPU idle: by default every warp then takes the dense kernel (8 warps per 32
// particles).  StepConsts::dense_window / dense_all override the defaults
// (pbf_autotune).
constexpr int kMaxFields = 6;                   // partial-sum fields of the largest pass
constexpr unsigned kFull = 0xffffffffu;
constexpr float kNormalMin = 1.17549435e-38f;  // the smallest normal float

// Whether every particle takes the dense kernel.
bool dense_for_all(const StepConsts& c, int n) { return c.dense_all >= 0 ? c.dense_all != 0 : n < kDenseAllBelow; }

enum PassKind { kLambda = 0, kDeltaP = 1, kDeltaPFinal = 2, kXsph = 3 };

// Everything any pass kernel needs (passed by value).
struct PassArgs {
  StepConsts c;
  Geometry G;
  const float4* X;        // positions the pass reads (sorted)
  const uint32_t* cs;     // cell prefix, cells + 1 entries
  int n;
  int counter;            // flags word holding this pass's dense-list length
  int next_counter;       // the other one, cleared for the next pass
  int item_counter;       // flags word handing out this pass's dense batches
  int next_item_counter;  // the other one, cleared for the next pass
  int dense_all;          // every warp takes the dense kernel (small n)
  uint32_t* flags;
  uint32_t* dense;
  // the positions by component (x at S, y at S + stride, z at S + 2 stride):
  // the sparse kernel's candidate tests read four at a time
  const float* S;
  float* S_out;           // delta_p: out, beside T / npos
  int stride;             // of S
  uint32_t* hits;         // hit lists: lambda writes them, delta_p reads them
  int* hit_n;
  int hit_stride;         // slots with a list
  uint32_t* cell_flags;   // CellFlag bits per cell
  const uint32_t* skeys;  // stale cell of each sorted slot
  float* lambda;          // lambda: out;  delta_p: in
  float4* XL;             // lambda: out, (position, lambda): the delta_p passes' X
  float* rho;             // lambda: out;  delta_p_final and xsph: in
  float4* T;              // delta_p: out
  float4* VR;             // (velocity, rho): delta_p_final: out;  xsph: in
  const float4* xs;       // delta_p_final: sorted x at t
  const uint32_t* iid_s;  // delta_p_final: sorted iid
  float4* npos;           // delta_p_final: out
  float4* vel;            // delta_p_final: out
  float4* pos;            // delta_p_final: out (permuted inputs)
  uint32_t* iid;          // delta_p_final: out (permuted inputs)
  const float4* V;        // xsph: velocities
  float4* NV;             // xsph: out
  // group tables (the dense kernel visits groups of grouped cells)
  const int* grp_off;
  const int* grp_n;
  const int* grp_cnt;
  const float4* grp_pos;
  const float4* grp_sum;
  const float4* grp_aux;
  // the particles the pass computes: list[0, flags[count_word]) (null: every
  // particle, in order); the work list of the lambda / delta_p passes, or the
  // current-cell buckets.  identity_word >= 0: a flag saying the list is the
  // identity (every particle in order)
  const int* list;
  int count_word;
  int identity_word;
  // the list is the buckets with every cell's on an even slot (pair_slots; an
  // empty slot holds -1): the sparse kernel of the lambda and xsph passes takes
  // the two slots of a pair in one thread
  int paired;
  int moved_word;         // delta_p: a flag counting the particles that left their grid cell (-1: none)
};

// The particle that thread slot t of a pass computes (t < work_count(a)).
__device__ __forceinline__ int work_count(const PassArgs& a) {
  return a.list ? (int)a.flags[a.count_word] : a.n;
}
__device__ __forceinline__ int work_particle(const PassArgs& a, int t) {
  return a.list && !(a.identity_word >= 0 && a.flags[a.identity_word]) ? __ldg(a.list + t) : t;
}

// Component copy of position x of particle i (PassArgs::S).
__device__ __forceinline__ void put_components(float* S, int stride, int i, float4 x) {
  S[i] = x.x;
  S[stride + i] = x.y;
  S[2 * (size_t)stride + i] = x.z;
}

// ---- windows ------------------------------------------------------------------------

// Sorted-slot range [s, e) of cells (x, y, z-1 .. z+1) clipped to the grid.
// cs[cells] == n, so e <= n; the clamps keep even an inconsistent table in range.
__device__ __forceinline__ void column_run(const SceneGeom& g, const uint32_t* __restrict__ cs,
                                           int n, int x, int y, int z, int& s, int& e) {
  const int zlo = max(z - 1, 0), zhi = min(z + 1, g.dims[2] - 1);
  const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
  s = (int)__ldg(cs + base + zlo);
  e = max(min((int)__ldg(cs + base + zhi + 1), n), s);
}

__device__ __forceinline__ int window_total(const SceneGeom& g, const uint32_t* __restrict__ cs,
                                            int n, int3 q) {
  int total = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      total += e - s;
    }
  }
  return total;
}

// Whether a cell of the window carries any of `bits`.  No branch in it and none
// around its loads: a cell outside the grid is read as the nearest one inside,
// which the window holds as well.  The loops with early exits that stood here
// let a warp's lanes leave one by one, and k_dense's barrier after them did not
// wait for the last ones (a part sum or a run of the block's previous batch was
// then read in place of this one's: 2 to 4 of 100 runs of four steps of 30,011 scattered particles).
__device__ __forceinline__ bool window_flagged(const SceneGeom& g,
                                               const uint32_t* __restrict__ cell_flags, int3 q,
                                               uint32_t bits) {
  uint32_t any = 0u;
#pragma unroll 1  // (nine loads in flight; all 27 cost the paired kernel registers)
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = min(max(q.x + dx, 0), g.dims[0] - 1);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int y = min(max(q.y + k / 3 - 1, 0), g.dims[1] - 1), z = min(max(q.z + k % 3 - 1, 0), g.dims[2] - 1);
      any |= cell_flags[cell_index(g, x, y, z)];
    }
  }
  return (any & bits) != 0u;
}

// ---- where a pass reads candidate positions ---------------------------------------------
//
// From global memory (X[j], read-only path), or from the block's staged copy
// of its window in shared memory.  Run r = 3 (dx + 1) + (dy + 1) of a window
// is one column of three z-consecutive cells; a block stages, per run, the
// slots of the z-range its particles' runs cover, and slot j of run r sits at
// S[j + D[r]].  Either source gives bitwise the same positions, so a pass's
// sums do not depend on which one it read.
struct FromGlobal {
  const float4* __restrict__ X;
  __device__ __forceinline__ float4 at(int j, int) const { return __ldg(X + j); }
  // hit-queue entry of a chunk starting at slot j of run r, and back
  __device__ __forceinline__ int tag(int j, int) const { return j; }
  __device__ __forceinline__ float4 untag(int t, int bit, int& j) const {
    j = t + bit;
    return __ldg(X + j);
  }
};

struct FromStage {
  const float4* S;  // shared memory: the staged runs
  const int* D;     // shared memory: per run, staged index - slot
  __device__ __forceinline__ float4 at(int j, int r) const { return S[j + D[r]]; }
  // staged index (< 2^16) and run
  __device__ __forceinline__ int tag(int j, int r) const { return (j + D[r]) | (r << 16); }
  __device__ __forceinline__ float4 untag(int t, int bit, int& j) const {
    const int v = (t & 0xffff) + bit;
    j = v - D[t >> 16];
    return S[v];
  }
};

// Every candidate of the window, in order.
template <class P, class Src>
__device__ __forceinline__ void visit_window(const SceneGeom& g, const uint32_t* __restrict__ cs,
                                             int n, int3 q, const Src& src, P& p) {
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int r = 3 * (dx + 1) + (dy + 1);
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      for (int j = s; j < e; ++j) p.visit(src.at(j, r), j);
    }
  }
}

// ---- hit queue ------------------------------------------------------------------------
//
// The masked walks below test a chunk of up to 32 consecutive candidates at a
// time into a bit mask (cheap, every lane busy) and run the pair body on the
// set bits only.  Running the body right after each chunk costs a warp
// max-over-lanes(hits of that chunk) body iterations per chunk; lanes whose
// particle has fewer hits in that chunk idle, chunk after chunk.  Instead each
// thread queues its non-empty chunks (mask + where the chunk starts) in shared
// memory and HitQueue::flush runs the body once per queued hit in one flat
// loop, so the warp pays max-over-lanes of the hits of the whole queued span.
// Hits are visited in the order they were queued -- the window's visiting
// order -- so the sums are bitwise those of visiting each chunk's hits right
// away.  The dense kernel's capacity (chunks queued per thread before a flush)
// comes from the step's tuning (StepConsts::queue_dense); capacity 1 runs
// each chunk's hits right away, straight from registers.  The sparse kernel
// has a queue of its own (QueueColumn).
struct HitQueue {
  uint32_t* mask;  // this thread's column: entry k at mask[k * stride]
  int* base;       // where queued chunk k starts (Src::tag)
  int stride;
  int cap;
  int n = 0;

  __device__ HitQueue(uint32_t* mask_, int* base_, int stride_, int cap_)
      : mask(mask_), base(base_), stride(stride_), cap(cap_) {}
  template <class P, class Src>
  __device__ __forceinline__ void flush(const Src& src, P& p) {
    uint32_t m = 0u;
    int b = 0, k = 0;
    for (;;) {
      if (!m) {
        if (k == n) break;
        m = mask[k * stride];  // every queued mask has a bit set
        b = base[k * stride];
        ++k;
      }
      const int bit = __ffs(m) - 1;
      m &= m - 1u;
      int j;
      const float4 xj = src.untag(b, bit, j);
      p.visit(xj, j);
    }
    n = 0;
  }
  template <class P, class Src>
  __device__ __forceinline__ void push(uint32_t m, int tag, const Src& src, P& p) {
    if (cap == 1) {  // no queue: the chunk's hits right away, straight from registers
      while (m) {
        const int bit = __ffs(m) - 1;
        m &= m - 1u;
        int j;
        const float4 xj = src.untag(tag, bit, j);
        p.visit(xj, j);
      }
      return;
    }
    if (!m) return;
    mask[n * stride] = m;
    base[n * stride] = tag;
    if (++n == cap) flush(src, p);
  }
};

// Hit mask of candidates [jb, jb + min(32, j1 - jb)) of run r (four loads in flight).
template <class P, class Src>
__device__ __forceinline__ uint32_t chunk_mask(const Src& src, int jb, int j1, int r, const P& p) {
  const int m = min(32, j1 - jb);
  uint32_t mask = 0u;
  int k = 0;
  for (; k + 3 < m; k += 4) {
    const float4 a = src.at(jb + k, r), b = src.at(jb + k + 1, r), c2 = src.at(jb + k + 2, r),
                 d = src.at(jb + k + 3, r);
    mask |= (uint32_t)p.hit(a, jb + k) << k;
    mask |= (uint32_t)p.hit(b, jb + k + 1) << (k + 1);
    mask |= (uint32_t)p.hit(c2, jb + k + 2) << (k + 2);
    mask |= (uint32_t)p.hit(d, jb + k + 3) << (k + 3);
  }
  for (; k < m; ++k) mask |= (uint32_t)p.hit(src.at(jb + k, r), jb + k) << k;
  return mask;
}

// Candidates [j0, j1) of run r, in order: with skip_misses (the pass's exact
// rules do not need every candidate) a hit mask per chunk of 32 (four loads in
// flight), its hits queued for p.visit() (the caller flushes hq); else every
// candidate, four loads in flight, after flushing what is queued.  Same result
// as visiting each candidate in turn.
template <class P, class Src>
__device__ __forceinline__ void visit_run(const Src& src, int j0, int j1, int r, P& p, bool skip_misses,
                                          HitQueue& hq) {
  if (skip_misses) {
    for (int jb = j0; jb < j1; jb += 32) hq.push(chunk_mask(src, jb, j1, r, p), src.tag(jb, r), src, p);
  } else {
    hq.flush(src, p);
    int j = j0;
    for (; j + 3 < j1; j += 4) {
      const float4 q0 = src.at(j, r), q1 = src.at(j + 1, r), q2 = src.at(j + 2, r), q3 = src.at(j + 3, r);
      p.visit(q0, j);
      p.visit(q1, j + 1);
      p.visit(q2, j + 2);
      p.visit(q3, j + 3);
    }
    for (; j < j1; ++j) p.visit(src.at(j, r), j);
  }
}

// Every candidate of the window, in order: a hit mask per chunk of 32
// consecutive slots of a run, p.visit() on the set bits.  p.visit() leaves
// non-hits untouched, so the result is that of visit_window.
template <class P, class Src>
__device__ __forceinline__ void visit_window_masked(const SceneGeom& g, const uint32_t* __restrict__ cs, int n,
                                                    int3 q, const Src& src, P& p, HitQueue& hq) {
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int r = 3 * (dx + 1) + (dy + 1);
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      visit_run(src, s, e, r, p, true, hq);
    }
  }
  hq.flush(src, p);
}

// Candidates [v_lo, v_hi) of the window (numbered in visiting order), run by
// run through visit_run (hit masks and the hit queue, or every candidate on
// the exact path).  The caller flushes hq.
template <class P, class Src>
__device__ __forceinline__ void visit_window_chunk(const SceneGeom& g, const uint32_t* __restrict__ cs, int n,
                                                   int3 q, const Src& src, P& p, int v_lo, int v_hi, HitQueue& hq) {
  int v0 = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int r = 3 * (dx + 1) + (dy + 1);
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      const int len = e - s;
      const int a = max(v_lo, v0), b = min(v_hi, v0 + len);
      if (a < b) visit_run(src, s + (a - v0), s + (b - v0), r, p, p.skip_misses(), hq);
      v0 += len;
    }
  }
  hq.flush(src, p);
}

// Part `part` of `parts` (a power of two) of the window, interleaved: the
// window's chunks of up to 32 consecutive candidates (per run, in visiting
// order) are numbered 0, 1, 2, ..., and chunk c belongs to part c mod parts.
// Parts of a window then hold about equal shares of its near and far
// candidates, so the warps that split a window finish together.  The caller
// flushes nothing: hq is flushed here.
template <class P, class Src>
__device__ __forceinline__ void visit_window_strided(const SceneGeom& g, const uint32_t* __restrict__ cs, int n,
                                                     int3 q, const Src& src, P& p, int part, int parts,
                                                     HitQueue& hq) {
  int c0 = 0;  // chunks of the window before this run
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int r = 3 * (dx + 1) + (dy + 1);
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      const int nch = (e - s + 31) >> 5;
      for (int k = (part - c0) & (parts - 1); k < nch; k += parts) {
        const int jb = s + 32 * k;
        visit_run(src, jb, min(jb + 32, e), r, p, p.skip_misses(), hq);
      }
      c0 += nch;
    }
  }
  hq.flush(src, p);
}

// Groups of cell `cell` in the pass's table, or -1 when the cell is visited
// particle by particle.
__device__ __forceinline__ int cell_groups(const PassArgs& a, int cell, int& slot) {
  const uint32_t sl = __ldg(a.cell_flags + cell) >> kCellSlotShift;
  slot = (int)sl - 1;
  return sl ? __ldg(a.grp_n + slot) : -1;
}

// Entries of the window when grouped cells count their groups.
__device__ __forceinline__ int window_total_grouped(const SceneGeom& g, const PassArgs& a, int3 q) {
  const int zlo = max(q.z - 1, 0), zhi = min(q.z + 1, g.dims[2] - 1);
  int total = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
      for (int z = zlo; z <= zhi; ++z) {
        int slot;
        const int ng = cell_groups(a, base + z, slot);
        if (ng > 0) {
          total += ng;
        } else {
          const int s0 = (int)__ldg(a.cs + base + z);
          total += max(min((int)__ldg(a.cs + base + z + 1), a.n), s0) - s0;
        }
      }
    }
  }
  return total;
}

// Entries [v_lo, v_hi) of the window in visiting order, grouped cells
// contributing their groups (p.visit_group; `own`: i belongs to the cell) and
// the other cells their particles (p.visit).  Without grouped cells this
// visits exactly what visit_window_chunk does, in the same order.
template <class P, class Src>
__device__ __forceinline__ void visit_window_grouped(const SceneGeom& g, const PassArgs& a, int3 q,
                                                     const Src& src, P& p, int v_lo, int v_hi, HitQueue& hq) {
  const int zlo = max(q.z - 1, 0), zhi = min(q.z + 1, g.dims[2] - 1);
  int v0 = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      const int r = 3 * (dx + 1) + (dy + 1);
      const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
      for (int z = zlo; z <= zhi; ++z) {
        int slot;
        const int ng = cell_groups(a, base + z, slot);
        const int s0 = (int)__ldg(a.cs + base + z);
        const int e0 = max(min((int)__ldg(a.cs + base + z + 1), a.n), s0);
        const int len = ng > 0 ? ng : e0 - s0;
        const int lo = max(v_lo, v0), hi = min(v_hi, v0 + len);
        if (lo < hi) {
          if (ng > 0) {
            hq.flush(src, p);  // queued hits come first in visiting order
            const int t0 = __ldg(a.grp_off + slot);
            const bool own = p.i >= s0 && p.i < e0;  // i is one of the cell's particles
            int t = t0 + (lo - v0);
            const int tend = t0 + (hi - v0);
            constexpr int U = P::kGroupUnroll;  // groups' loads in flight (unused parts are not loaded)
            for (; t + U - 1 < tend; t += U) {
              float4 gp[U], gs[U], ga[U];
              int gc[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                gp[u] = __ldg(a.grp_pos + t + u);
                gc[u] = __ldg(a.grp_cnt + t + u);
                gs[u] = __ldg(a.grp_sum + t + u);
                ga[u] = __ldg(a.grp_aux + t + u);
              }
#pragma unroll
              for (int u = 0; u < U; ++u) p.visit_group(gp[u], gc[u], gs[u], ga[u], own);
            }
            for (; t < tend; ++t)
              p.visit_group(__ldg(a.grp_pos + t), __ldg(a.grp_cnt + t), __ldg(a.grp_sum + t),
                            __ldg(a.grp_aux + t), own);
          } else {
            visit_run(src, s0 + (lo - v0), s0 + (hi - v0), r, p, p.skip_misses(), hq);
          }
        }
        v0 += len;
      }
    }
  }
  hq.flush(src, p);
}

// ---- the passes: per-candidate visit, partial-sum fields, finish ----------------------

// rsqrtf of a normal number (bitwise the same there, without the scaling of
// subnormal arguments; a zero gives +inf).
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct LambdaPass {
  static constexpr int kFields = 5;
  static constexpr int kGroupUnroll = 2;
  const StepConsts& c;
  const SceneGeom& g;
  float4 xi;
  int i;
  float pho = 0.f, gx = 0.f, gy = 0.f, gz = 0.f, gl2 = 0.f;

  __device__ LambdaPass(const PassArgs& a, const SceneGeom& g_, float4 xi_, int i_, bool)
      : c(a.c), g(g_), xi(xi_), i(i_) {}
  // candidates outside the cutoff add nothing (no exact rule in this pass)
  __device__ __forceinline__ bool skip_misses() const { return true; }
  __device__ __forceinline__ bool hit(float4 xj, int) const {
    return !(dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z) >= c.h2);
  }
  __device__ __forceinline__ void visit(float4 xj, int j) {
    const float ex = xi.x - xj.x, ey = xi.y - xj.y, ez = xi.z - xj.z;
    const float r2 = dist2(ex, ey, ez);
    if (!(r2 >= c.h2)) pair(ex, ey, ez, r2, j);  // NaN-inclusive, as getPoly6
  }
  __device__ __forceinline__ void pair(float ex, float ey, float ez, float r2, int j) {
    pho += poly6_inside(c, r2);
    if (!(r2 < c.keps2)) {  // as getSpikyGrad's |r| < KERNAL_EPS test
      const float ir = rsqrtf(r2);
      const float t = c.h - r2 * ir;
      const float sc = c.spiky_coef_rho0 * t * t * ir;
      const float ax = sc * ex, ay = sc * ey, az = sc * ez;
      gx += ax;
      gy += ay;
      gz += az;
      if (j != i) gl2 += dist2(ax, ay, az);
    }
  }
  // Two particles at r2 < h2, a then b (b only if `two`), keps2 > 0: pair() of
  // each.  Below keps2 (i itself among them) the gradient's factor is zero,
  // which adds nothing to the sums.
  __device__ __forceinline__ void visit_two(float4 xa, float4 xb, float4, float4, bool two) {
    const f32x2 ex = sub2(both(xi.x), pack2(xa.x, xb.x)), ey = sub2(both(xi.y), pack2(xa.y, xb.y)),
                ez = sub2(both(xi.z), pack2(xa.z, xb.z));
    const f32x2 r2 = dist2_2(ex, ey, ez);
    float ra, rb;
    unpack2(r2, ra, rb);
    const f32x2 d = sub2(both(c.h2), r2);
    const f32x2 w = mul2(mul2(both(c.poly6_coef), d), d);
    const f32x2 ir = pack2(rsqrt_normal(ra), rsqrt_normal(rb));
    const f32x2 t = fma2(r2, ir, both(-c.h));  // -(h - |r|); its sign cancels in t t
    const f32x2 scu = mul2(mul2(mul2(both(c.spiky_coef_rho0), t), t), ir);
    float sa, sb, wa, wb, da, db;
    unpack2(scu, sa, sb);
    unpack2(w, wa, wb);
    unpack2(d, da, db);
    sa = ra < c.keps2 ? 0.f : sa;
    sb = rb < c.keps2 || !two ? 0.f : sb;
    wb = two ? wb : 0.f;
    const f32x2 sc = pack2(sa, sb);
    const f32x2 ax = mul2(sc, ex), ay = mul2(sc, ey), az = mul2(sc, ez);
    const f32x2 l = dist2_2(ax, ay, az);
    float xa_, xb_, ya_, yb_, za_, zb_, la, lb;
    unpack2(l, la, lb);
    pho = fmaf(wa, da, pho);
    pho = fmaf(wb, db, pho);
    unpack2(ax, xa_, xb_), unpack2(ay, ya_, yb_), unpack2(az, za_, zb_);
    gx += xa_, gy += ya_, gz += za_;
    gx += xb_, gy += yb_, gz += zb_;
    gl2 += la;
    gl2 += lb;
  }
  // `cnt` particles at xg.  The group holding i itself lies at r2 = 0 <
  // keps2 (grouping needs keps2 > 0): no gradient, as the reference's j != i.
  __device__ __forceinline__ void visit_group(float4 xg, int cnt, float4, float4, bool) {
    const float ex = xi.x - xg.x, ey = xi.y - xg.y, ez = xi.z - xg.z;
    const float r2 = dist2(ex, ey, ez);
    if (!(r2 >= c.h2)) {
      const float fc = (float)cnt;
      pho += fc * poly6_inside(c, r2);
      if (!(r2 < c.keps2)) {
        const float ir = rsqrtf(r2);
        const float t = c.h - r2 * ir;
        const float sc = c.spiky_coef_rho0 * t * t * ir;
        const float ax = sc * ex, ay = sc * ey, az = sc * ez;
        gx += fc * ax;
        gy += fc * ay;
        gz += fc * az;
        gl2 += fc * dist2(ax, ay, az);
      }
    }
  }
  __device__ void store(float* f, int stride) const {
    f[0] = pho, f[stride] = gx, f[2 * stride] = gy, f[3 * stride] = gz, f[4 * stride] = gl2;
  }
  __device__ void add(const float* f, int stride) {
    pho += f[0], gx += f[stride], gy += f[2 * stride], gz += f[3 * stride], gl2 += f[4 * stride];
  }
  __device__ void finish(const PassArgs& a) const {
    float rho = pho;
    if (c.k_b != 0.f) rho += c.k_b * boundary_density(c, g, xi);
    const float grad_l2 = gl2 + dist2(gx, gy, gz);
    const float lam = -(rho / c.pho0 - 1.f) / (grad_l2 + c.lambda_eps);
    a.lambda[i] = lam;
    a.rho[i] = rho;
    a.XL[i] = make_float4(xi.x, xi.y, xi.z, lam);
    const uint32_t bits = (isfinite(lam) ? 0u : (uint32_t)kCellLambdaNonFinite) |
                          (rho > 0.f && isfinite(rho) ? 0u : (uint32_t)kCellRhoNotPositive);
    if (bits) {
      atomicOr(&a.cell_flags[a.skeys[i]], bits);
      if (bits & kCellLambdaNonFinite) atomicOr(&a.flags[kFlagLambdaNonFinite], 1u);
      if (bits & kCellRhoNotPositive) atomicOr(&a.flags[kFlagXsphExact], 1u);
    }
  }
};

// sum over neighbours j != i of (lambda_i + lambda_j + s_corr) grad W.  exact
// adds the reference's poisoning of the sum by a non-finite lambda through a
// zero gradient (candidates j != i outside the cutoff).
template <bool kFinal>
struct DeltaPPass {
  static constexpr int kFields = 4;
  static constexpr int kGroupUnroll = 2;
  const StepConsts& c;
  const SceneGeom& g;
  float4 xi;  // positions come with their lambda in w (PassArgs::XL)
  int i;
  float li;
  bool exact;
  float ax = 0.f, ay = 0.f, az = 0.f;
  bool poison = false;

  __device__ DeltaPPass(const PassArgs& a, const SceneGeom& g_, float4 xi_, int i_, bool exact_)
      : c(a.c), g(g_), xi(xi_), i(i_), li(xi_.w), exact(exact_) {}
  __device__ __forceinline__ bool skip_misses() const { return !exact; }
  __device__ __forceinline__ bool hit(float4 xj, int j) const {
    const float r2 = dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
    return !(r2 >= c.h2) && !(r2 < c.keps2) && j != i;
  }
  __device__ __forceinline__ void visit(float4 xj, int j) {
    const float ex = xi.x - xj.x, ey = xi.y - xj.y, ez = xi.z - xj.z;
    const float r2 = dist2(ex, ey, ez);
    if (!(r2 >= c.h2) && !(r2 < c.keps2) && j != i) {  // NaN-inclusive, as the reference
      pair(ex, ey, ez, r2, xj.w);
    } else if (exact && j != i) {
      // zero gradient: (lambda_i + lambda_j + s_corr) * 0 is NaN iff a lambda is not finite
      poison |= !isfinite(li) || !isfinite(xj.w);
    }
  }
  // Two particles at r2 < h2, a then b, keps2 > 0, not on the exact path:
  // pair() of each.  Below keps2 (i itself among them) the factor is zero,
  // which adds nothing to the sums.
  __device__ __forceinline__ void visit_two(float4 xa, float4 xb, float4, float4, bool two) {
    const f32x2 ex = sub2(both(xi.x), pack2(xa.x, xb.x)), ey = sub2(both(xi.y), pack2(xa.y, xb.y)),
                ez = sub2(both(xi.z), pack2(xa.z, xb.z));
    const f32x2 r2 = dist2_2(ex, ey, ez);
    float ra, rb;
    unpack2(r2, ra, rb);
    const f32x2 d = sub2(both(c.h2), r2);
    const f32x2 w = mul2(mul2(mul2(both(c.poly6_coef), d), d), d);
    f32x2 pw;
    if (c.npow == 4) {
      const f32x2 w2 = mul2(w, w);
      pw = mul2(w2, w2);
    } else {
      float wa, wb;
      unpack2(w, wa, wb);
      pw = pack2(pow_corr(c, wa), pow_corr(c, wb));
    }
    const f32x2 ll = add2(both(li), pack2(xa.w, xb.w));
    const f32x2 lc = fma2(both(c.coef_corr), pw, ll);
    const f32x2 ir = pack2(rsqrt_normal(ra), rsqrt_normal(rb));
    const f32x2 t = fma2(r2, ir, both(-c.h));  // -(h - |r|); its sign cancels in t t
    const f32x2 f = mul2(lc, mul2(mul2(mul2(both(c.spiky_coef), t), t), ir));
    float fa, fb, xa_, xb_, ya_, yb_, za_, zb_;
    unpack2(f, fa, fb);
    fa = ra < c.keps2 ? 0.f : fa;
    fb = rb < c.keps2 || !two ? 0.f : fb;
    unpack2(ex, xa_, xb_), unpack2(ey, ya_, yb_), unpack2(ez, za_, zb_);
    ax = fmaf(fa, xa_, ax), ay = fmaf(fa, ya_, ay), az = fmaf(fa, za_, az);
    ax = fmaf(fb, xb_, ax), ay = fmaf(fb, yb_, ay), az = fmaf(fb, zb_, az);
  }
  __device__ __forceinline__ void pair(float ex, float ey, float ez, float r2, float lj) {
    const float wgt = poly6_inside(c, r2);
    const float corr = c.coef_corr * pow_corr(c, wgt);
    const float ir = rsqrtf(r2);
    const float t = c.h - r2 * ir;
    const float f = (li + lj + corr) * (c.spiky_coef * t * t * ir);
    ax = fmaf(f, ex, ax);
    ay = fmaf(f, ey, ay);
    az = fmaf(f, ez, az);
  }
  // `cnt` particles at xg with lambda_j summing to cnt sum.x + sum.y (each
  // lambda_j - sum.x finite, or lambda_j the same bits as sum.x).  exact: the
  // poisoning rule for the group's members j != i (i is a member when it
  // belongs to the cell and sits at xg).
  __device__ __forceinline__ void visit_group(float4 xg, int cnt, float4 sum, float4, bool own) {
    const float ex = xi.x - xg.x, ey = xi.y - xg.y, ez = xi.z - xg.z;
    const float r2 = dist2(ex, ey, ez);
    if (!(r2 >= c.h2) && !(r2 < c.keps2)) {
      const float wgt = poly6_inside(c, r2);
      const float corr = c.coef_corr * pow_corr(c, wgt);
      const float ir = rsqrtf(r2);
      const float t = c.h - r2 * ir;
      const float f = ((float)cnt * (li + sum.x + corr) + sum.y) * (c.spiky_coef * t * t * ir);
      ax = fmaf(f, ex, ax);
      ay = fmaf(f, ey, ay);
      az = fmaf(f, ez, az);
    } else if (exact) {
      const bool member = own && __float_as_uint(xi.x) == __float_as_uint(xg.x) &&
                          __float_as_uint(xi.y) == __float_as_uint(xg.y) &&
                          __float_as_uint(xi.z) == __float_as_uint(xg.z);
      if (cnt > (member ? 1 : 0)) poison |= !isfinite(li) || !isfinite(sum.x);
    }
  }
  __device__ void store(float* f, int stride) const {
    f[0] = ax, f[stride] = ay, f[2 * stride] = az, f[3 * stride] = poison ? 1.f : 0.f;
  }
  __device__ void add(const float* f, int stride) {
    ax += f[0], ay += f[stride], az += f[2 * stride];
    poison |= f[3 * stride] != 0.f;
  }
  // d / pho0, per-component clamp to +-max_dp, wall clamp
  // (fluids/Simulator_kernel.cuh:184-193); fminf/fmaxf map a NaN to the bound.
  __device__ void finish(const PassArgs& a) const {
    float sx = ax, sy = ay, sz = az;
    if (poison) sx = sy = sz = __int_as_float(0x7fffffff);
    const float dx = fmaxf(fminf(sx / c.pho0, c.max_dp), -c.max_dp);
    const float dy = fmaxf(fminf(sy / c.pho0, c.max_dp), -c.max_dp);
    const float dz = fmaxf(fminf(sz / c.pho0, c.max_dp), -c.max_dp);
    const float4 xf = make_float4(fmaxf(fminf(xi.x + dx, g.hi[0]), g.lo[0]),
                                  fmaxf(fminf(xi.y + dy, g.hi[1]), g.lo[1]),
                                  fmaxf(fminf(xi.z + dz, g.hi[2]), g.lo[2]), 0.f);
    put_components(a.S_out, a.stride, i, xf);
    if (a.moved_word >= 0) {  // how many leave their grid cell
      const int3 q = cell_of(c, g, xf);
      const bool moved = (uint32_t)cell_index(g, q.x, q.y, q.z) != a.skeys[i];
      const unsigned act = __activemask(), left = __ballot_sync(act, moved);
      if (left && (threadIdx.x & 31) == __ffs(act) - 1) atomicAdd(&a.flags[a.moved_word], (uint32_t)__popc(left));
    }
    if (!kFinal) {
      a.T[i] = xf;
      return;
    }
    // last iteration: x_final -> npos, v = (x_final - x) * (1/dt) -> vel, and the
    // caller's pos / iid receive the permuted inputs (the reference's in-place sort)
    const float4 x0 = a.xs[i];
    a.npos[i] = make_float4(xf.x, xf.y, xf.z, x0.w);
    const float4 v = make_float4((xf.x - x0.x) * c.inv_dt, (xf.y - x0.y) * c.inv_dt,
                                 (xf.z - x0.z) * c.inv_dt, 0.f);
    a.vel[i] = v;
    a.VR[i] = make_float4(v.x, v.y, v.z, a.rho[i]);
    if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z)) {
      atomicOr(&a.cell_flags[a.skeys[i]], (uint32_t)kCellVelNonFinite);
      atomicOr(&a.flags[kFlagXsphExact], 1u);
    }
    a.pos[i] = x0;
    a.iid[i] = a.iid_s[i];
  }
};

// sum over the window of 2 (v_j - v_i) W / (rho_i + rho_j).  exact adds the
// reference's NaN from 0 * v / (rho_i + rho_j) outside the cutoff.
struct XsphPass {
  static constexpr int kFields = 6;
  static constexpr int kGroupUnroll = 2;
  const StepConsts& c;
  const float4* __restrict__ VR;  // (velocity, rho)
  float4 xi, vi;
  float ri;
  int i;
  bool exact;
  float ax = 0.f, ay = 0.f, az = 0.f;
  bool px = false, py = false, pz = false;

  __device__ XsphPass(const PassArgs& a, const SceneGeom&, float4 xi_, int i_, bool exact_)
      : c(a.c), VR(a.VR), xi(xi_), vi(a.VR[i_]), ri(vi.w), i(i_), exact(exact_) {}
  __device__ __forceinline__ bool skip_misses() const { return !exact; }
  __device__ __forceinline__ bool hit(float4 xj, int) const {
    return !(dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z) >= c.h2);
  }
  __device__ __forceinline__ void visit(float4 xj, int j) {
    // v_j and rho_j first: their load overlaps the distance test (a visited
    // candidate is almost always a neighbour)
    const float4 vj = __ldg(VR + j);
    const float r2 = dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
    if (!(r2 >= c.h2)) {  // NaN-inclusive, as getPoly6
      pair(vj, r2);
    } else if (exact) {
      miss(vj);
    }
  }
  // A candidate outside the cutoff (W = 0): 2 (v_j - v_i) * 0 / (rho_i + rho_j) is
  // NaN iff the velocity difference is not finite or the denominator is 0 or NaN.
  __device__ __forceinline__ void miss(float4 vj) {
    const float den = ri + vj.w;
    const bool bad_den = !(den != 0.f) || isnan(den);
    px |= bad_den || !isfinite(vj.x - vi.x);
    py |= bad_den || !isfinite(vj.y - vi.y);
    pz |= bad_den || !isfinite(vj.z - vi.z);
  }
  // miss() for a candidate outside the cutoff.
  __device__ __forceinline__ void miss_beyond(float4 xj, float4 vj) {
    if (dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z) >= c.h2) miss(vj);
  }
  // Two particles at r2 < h2, a then b (b only if `two`), not on the exact path.
  __device__ __forceinline__ void visit_two(float4 xa, float4 xb, float4 va, float4 vb, bool two) {
    pair(va, dist2(xi.x - xa.x, xi.y - xa.y, xi.z - xa.z));
    if (two) pair(vb, dist2(xi.x - xb.x, xi.y - xb.y, xi.z - xb.z));
  }
  __device__ __forceinline__ void pair(float4 vj, float r2) {
    const float w2 = 2.f * poly6_inside(c, r2) / (ri + vj.w);
    ax = fmaf(vj.x - vi.x, w2, ax);
    ay = fmaf(vj.y - vi.y, w2, ay);
    az = fmaf(vj.z - vi.z, w2, az);
  }
  // `cnt` particles at xg sharing the density sum.w and the velocity aux.xyz
  // (sum.xyz: the sum over the group of v_j - aux.xyz, zero for the groups
  // built here).
  // exact: the rule for 0 * (v_j - v_i) / (rho_i + rho_j) outside the cutoff;
  // the group build guarantees that every member's v_j - aux is finite or
  // that v_j is aux itself, so the first member's velocity decides.
  __device__ __forceinline__ void visit_group(float4 xg, int cnt, float4 sum, float4 aux, bool) {
    const float r2 = dist2(xi.x - xg.x, xi.y - xg.y, xi.z - xg.z);
    if (!(r2 >= c.h2)) {
      const float fc = (float)cnt;
      const float w2 = 2.f * poly6_inside(c, r2) / (ri + sum.w);
      ax = fmaf(fmaf(fc, aux.x - vi.x, sum.x), w2, ax);
      ay = fmaf(fmaf(fc, aux.y - vi.y, sum.y), w2, ay);
      az = fmaf(fmaf(fc, aux.z - vi.z, sum.z), w2, az);
    } else if (exact) {
      const float den = ri + sum.w;
      const bool bad_den = !(den != 0.f) || isnan(den);
      px |= bad_den || !isfinite(aux.x - vi.x);
      py |= bad_den || !isfinite(aux.y - vi.y);
      pz |= bad_den || !isfinite(aux.z - vi.z);
    }
  }
  __device__ void store(float* f, int stride) const {
    f[0] = ax, f[stride] = ay, f[2 * stride] = az;
    f[3 * stride] = px ? 1.f : 0.f, f[4 * stride] = py ? 1.f : 0.f, f[5 * stride] = pz ? 1.f : 0.f;
  }
  __device__ void add(const float* f, int stride) {
    ax += f[0], ay += f[stride], az += f[2 * stride];
    px |= f[3 * stride] != 0.f, py |= f[4 * stride] != 0.f, pz |= f[5 * stride] != 0.f;
  }
  __device__ void finish(const PassArgs& a) const {
    const float qnan = __int_as_float(0x7fffffff);
    a.NV[i] = make_float4(fmaf(c.c_xsph, px ? qnan : ax, vi.x), fmaf(c.c_xsph, py ? qnan : ay, vi.y),
                          fmaf(c.c_xsph, pz ? qnan : az, vi.z), 0.f);
  }
};

template <int kKind> struct PassOf;
template <> struct PassOf<kLambda> { using type = LambdaPass; };
template <> struct PassOf<kDeltaP> { using type = DeltaPPass<false>; };
template <> struct PassOf<kDeltaPFinal> { using type = DeltaPPass<true>; };
template <> struct PassOf<kXsph> { using type = XsphPass; };

// Whether particle i must visit every candidate of its window to reproduce the
// reference's IEEE poisoning (a strict superset of the particles whose sums
// can be poisoned): only when the step raised the pass's flag and i's own
// values or a flagged cell of its window could poison its sum.
__device__ __forceinline__ bool exact_path(int kind, const PassArgs& a, const SceneGeom& g,
                                           int3 q, int i) {
  // (the flags are the same for every lane; the rest is evaluated without branches)
  if (kind == kDeltaP || kind == kDeltaPFinal) {
    if (a.flags[kFlagLambdaNonFinite] == 0u) return false;
    const bool own = !isfinite(a.lambda[i]);
    return own | window_flagged(g, a.cell_flags, q, kCellLambdaNonFinite);
  }
  if (kind == kXsph) {
    if (a.flags[kFlagXsphExact] == 0u) return false;
    const float ri = a.rho[i];
    const float4 vi = a.V[i];
    const bool own = !(ri > 0.f) | !isfinite(ri) | !isfinite(vi.x) | !isfinite(vi.y) | !isfinite(vi.z);
    return own | window_flagged(g, a.cell_flags, q, kCellRhoNotPositive | kCellVelNonFinite);
  }
  return false;
}

// Whether only a window's flagged cells can poison the xsph sum of a particle
// with this velocity and density: elsewhere 0 < rho_j, v_j is finite, and
// |v_j - v_i| then rounds to a finite number (kTameSpeed is below half a unit in
// the last place of the largest).
constexpr float kTameSpeed = 1e30f;
__device__ __forceinline__ bool tame(float4 vr) {
  return vr.w > 0.f && isfinite(vr.w) && fabsf(vr.x) < kTameSpeed && fabsf(vr.y) < kTameSpeed &&
         fabsf(vr.z) < kTameSpeed;
}

// ---- window staging: bulk async copies into shared memory ------------------------------
//
// With the passes taking particles in current-cell order, the particles of a
// block usually sit in cells of one column (scene, x, y), z-consecutive: their
// windows are then made of the same 9 column runs, each particle's run r a
// z-sub-range of the block's run r, which covers cells [zmin - 1, zmax + 1] of
// column (x + dx, y + dy) -- one contiguous range of sorted slots.  Such a
// block copies its runs' positions (16 bytes a slot, 16-byte aligned) into
// shared memory with one cp.async.bulk per run, all completing on one
// mbarrier, and its threads then walk their windows there (FromStage) instead
// of through L1 (FromGlobal).  Blocks whose particles span several columns,
// whose runs exceed the stage, or whose runs hold a grouped cell read global
// memory as before.  The wait is bounded: past kStageSpins polls the block
// records kErrStageTimeout, stops staging and reads global memory (same
// results), and waits once more (bounded) for the copy before it exits.
// On GB300 the staged variants measured slower than the L1 path on every
// workload tried (the candidates are L1-resident already, and the stage costs
// resident blocks and a wait per block), so the default stages are 0 and
// pbf_autotune turns them on only where its trial steps find them faster.

constexpr int kStageSpins = 1 << 20;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0u;
}
// Bounded wait for the phase of the given parity to complete.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  for (int k = 0; k < kStageSpins; ++k)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// bytes (a multiple of 16) from global src to shared dst (both 16-byte
// aligned), completing as transaction bytes on bar.  A CTA's own shared
// memory address is a valid shared::cluster address (no cluster launch, no
// multicast).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// Orders this thread's earlier generic-proxy accesses of shared memory (the
// previous item's reads of the stage) before its following async-proxy writes.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// A block's staging state in shared memory.
struct StageState {
  uint64_t bar;
  int D[9];           // per run: staged index - first slot
  int ok;             // this item's runs are staged
  int failed;         // a wait gave up: the block stages no more
  int wx[kDenseThreads / 32], wy[kDenseThreads / 32], wcb[kDenseThreads / 32];
  int wzmin[kDenseThreads / 32], wzmax[kDenseThreads / 32], wi[kDenseThreads / 32];
  int wsame[kDenseThreads / 32];
};

// Votes of one warp: whether its participating lanes share (scene, x, y), the
// z-range they cover and one participating particle (lane 0 of the warp writes
// st.w*[w]).  Every lane of the warp calls it.
__device__ __forceinline__ void stage_vote(StageState& st, int w, bool part, const SceneGeom& g, int3 q,
                                           int i) {
  const unsigned pm = __ballot_sync(kFull, part);
  const int lead = pm ? __ffs(pm) - 1 : 0;
  const int lx = __shfl_sync(kFull, q.x, lead), ly = __shfl_sync(kFull, q.y, lead);
  const int lcb = __shfl_sync(kFull, g.cell_base, lead), li = __shfl_sync(kFull, i, lead);
  const bool same = __all_sync(kFull, !part || (q.x == lx && q.y == ly && g.cell_base == lcb));
  const int zmin = __reduce_min_sync(kFull, part ? q.z : INT_MAX);
  const int zmax = __reduce_max_sync(kFull, part ? q.z : INT_MIN);
  if ((threadIdx.x & 31) == 0) {
    st.wsame[w] = pm == 0u ? -1 : (same ? 1 : 0);  // -1: no participating lane
    st.wx[w] = lx, st.wy[w] = ly, st.wcb[w] = lcb, st.wi[w] = li;
    st.wzmin[w] = zmin, st.wzmax[w] = zmax;
  }
}

// Thread 0, after the votes of warps [0, nw): when every participating lane
// shares one column and its runs fit in `cap` slots and hold no grouped cell,
// sets st.D, arms st.bar for the runs' bytes and issues one bulk copy per
// non-empty run into S; st.ok says whether it did.
__device__ __forceinline__ void stage_issue(StageState& st, int nw, const PassArgs& a, float4* S, int cap) {
  st.ok = 0;
  if (st.failed || cap <= 0) return;
  int w0 = -1, zmin = INT_MAX, zmax = INT_MIN;
  for (int w = 0; w < nw; ++w) {
    if (st.wsame[w] < 0) continue;
    if (st.wsame[w] == 0) return;
    if (w0 < 0) {
      w0 = w;
    } else if (st.wx[w] != st.wx[w0] || st.wy[w] != st.wy[w0] || st.wcb[w] != st.wcb[w0]) {
      return;
    }
    zmin = min(zmin, st.wzmin[w]);
    zmax = max(zmax, st.wzmax[w]);
  }
  if (w0 < 0) return;
  const SceneGeom g = geom_of(a.c, a.G, st.wi[w0]);
  const int x0 = st.wx[w0], y0 = st.wy[w0];
  const int zlo = max(zmin - 1, 0), zhi = min(zmax + 1, g.dims[2] - 1);
  const bool groups = a.flags[kGroupCount] != 0u;
  int s[9], e[9], total = 0;
  for (int r = 0; r < 9; ++r) {
    const int x = x0 + r / 3 - 1, y = y0 + r % 3 - 1;
    s[r] = e[r] = 0;
    if (x < 0 || x >= g.dims[0] || y < 0 || y >= g.dims[1]) continue;
    const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
    s[r] = (int)__ldg(a.cs + base + zlo);
    e[r] = max(min((int)__ldg(a.cs + base + zhi + 1), a.n), s[r]);
    total += e[r] - s[r];
    if (groups)
      for (int z = zlo; z <= zhi; ++z)
        if (__ldg(a.cell_flags + base + z) >> kCellSlotShift) return;  // a grouped cell
  }
  if (total > cap) return;
  fence_proxy_async_smem();
  mbar_arrive_expect_tx(&st.bar, (uint32_t)total * (uint32_t)sizeof(float4));
  int v = 0;
  for (int r = 0; r < 9; ++r) {
    st.D[r] = v - s[r];
    const int len = e[r] - s[r];
    if (len > 0) bulk_g2s(S + v, a.X + s[r], (uint32_t)len * (uint32_t)sizeof(float4), &st.bar);
    v += len;
  }
  st.ok = 1;
}

// Every thread, after stage_issue and a barrier: waits (bounded) for the
// staged runs.  Returns whether the item reads them; a wait that gave up
// (block-uniform through the barrier) records the error and stops staging.
__device__ __forceinline__ bool stage_wait(StageState& st, const PassArgs& a, uint32_t& phase) {
  if (!st.ok) return false;  // uniform: written before the barrier
  const bool done = mbar_wait_bounded(&st.bar, phase);
  const bool any_failed = __syncthreads_or(!done);
  if (any_failed) {
    if (threadIdx.x == 0) {
      st.failed = 1;
      atomicOr(&a.flags[kErrorWord], (uint32_t)kErrStageTimeout);
    }
    return false;  // st.failed is read only after the next barrier
  }
  phase ^= 1u;
  return true;
}

// Before a block that staged exits: a wait that gave up leaves its copy in
// flight, so wait once more (bounded) for it.
__device__ __forceinline__ void stage_drain(StageState& st, uint32_t phase) {
  if (threadIdx.x == 0 && st.failed) mbar_wait_bounded(&st.bar, phase);
}

// ---- kernels ------------------------------------------------------------------------

// The stage's barrier, before first use (thread 0).
__device__ __forceinline__ void stage_init(StageState& st) {
  st.failed = 0;
  st.ok = 0;
  mbar_init(&st.bar, 1u);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// ---- hits of a window -------------------------------------------------------------------
//
// The sparse kernel's walk.  Candidates are tested four at a time on the
// component copies of the positions (three 16-byte loads, two candidates to a
// packed float instruction, rounded as dist2 rounds), and the sign of r2 - h2
// is shifted into a hit mask, so a test costs no compare, no select and no
// branch.  Runs start anywhere, so the groups start at the run's start rounded
// down to four and the mask drops what lies outside the run.  Non-empty masks
// are queued in shared memory and one flat loop visits the window's hits at
// the end: a warp then iterates as often as its busiest lane has hits in the
// whole window (~42 at rest density for 33 on average), not the sum over the
// chunks of the busiest lane of each (~72).  Visiting order: slots ascending
// in each run, runs in order -- the reference's.  The visits take two hits at
// a time in packed arithmetic, rounded as pair() rounds them.
//
// This holds with kernel_eps a normal number (fast_hits) and for a particle at
// a finite position (a NaN one would meet itself); others take
// visit_window_masked.

// The sign bits of d, the lower half's first.
__device__ __forceinline__ uint32_t shift_in(uint32_t mask, f32x2 d) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(d));
  return __funnelshift_l(hi, __funnelshift_l(lo, mask, 1), 1);
}

// The component copies of candidates j .. j + 3 (j a multiple of 4).
struct Four {
  ulonglong2 x, y, z;
  __device__ __forceinline__ Four(const float* __restrict__ S, int stride, int j)
      : x(__ldg(reinterpret_cast<const ulonglong2*>(S + j))),
        y(__ldg(reinterpret_cast<const ulonglong2*>(S + stride + j))),
        z(__ldg(reinterpret_cast<const ulonglong2*>(S + 2 * (size_t)stride + j))) {}
};

// The window's centre, negated, and the largest float below h2, twice each:
// r2 is a hit when that minus r2 has no sign bit, i.e. when r2 < h2 or r2 is
// NaN (a NaN result has none), the reference's !(r2 >= h2).
struct HitTest {
  f32x2 x, y, z, h;
  __device__ __forceinline__ HitTest(float4 xi, float h2)
      : x(both(-xi.x)), y(both(-xi.y)), z(both(-xi.z)),
        h(both(below(h2))) {}
  static __device__ __forceinline__ float below(float h2) {
    return h2 > 0.f ? __uint_as_float(__float_as_uint(h2) - 1u) : -1.f;
  }
  __device__ __forceinline__ f32x2 pair(f32x2 px, f32x2 py, f32x2 pz) const {
    return sub2(h, dist2_2(add2(px, x), add2(py, y), add2(pz, z)));
  }
  // the four's miss bits shifted into mask
  __device__ __forceinline__ uint32_t four(const Four& f, uint32_t mask) const {
    mask = shift_in(mask, pair(f.x.x, f.y.x, f.z.x));
    return shift_in(mask, pair(f.x.y, f.y.y, f.z.y));
  }
};

// A thread's column of shared memory: the queue grows from entry 0, the
// window's runs [s, e) wait in entries kRunSlot.. until they are walked.
// Queue entry k: the chunk's mask and its first slot in run[k], and, where two
// particles share the walk, the second one's mask in second[k].
constexpr int kQueueSlots = 12;
constexpr int kRunSlot = kQueueSlots - 9;
struct QueueColumn {
  uint2* run;
  uint32_t* second;
};

// The hits of one particle in queue entries [0, n), one after the other; the
// caller counts them.
template <bool kSecond, int kStride>
struct QueuedHits {
  QueueColumn q;
  uint32_t m = 0u;
  int base = 0;
  __device__ __forceinline__ explicit QueuedHits(QueueColumn q_) : q(q_) {}
  __device__ __forceinline__ int next() {
    while (!m) {  // (an entry of a pair may hold hits of the other particle only)
      if (kSecond) {
        m = *q.second;
        base = (int)q.run->y;
      } else {
        const uint2 e = *q.run;
        m = e.x;
        base = (int)e.y;
      }
      q.run += kStride;
      q.second += kStride;
    }
    const int bit = __clz(m);  // the first candidate is the highest bit
    m ^= 0x80000000u >> bit;
    return base + bit;
  }
};

// Visits `hits` queued hits in order, two at a time, each two's loads issued
// two ahead.  out: where the lambda pass lists them (null: nowhere).
template <int kKind, bool kSecond, int kStride, class P>
__device__ __forceinline__ void visit_queued(const PassArgs& a, QueueColumn q, int hits, P& p, uint32_t* out) {
  if (hits == 0) return;
  QueuedHits<kSecond, kStride> h(q);
  float4 xa, xb, va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
  // the next two hits (the second one the first again when only one is left)
  auto fetch = [&](int left) {
    const int ja = h.next(), jb = left > 1 ? h.next() : ja;
    xa = __ldg(a.X + ja);
    xb = __ldg(a.X + jb);
    if constexpr (kKind == kXsph) {
      va = __ldg(a.VR + ja);
      vb = __ldg(a.VR + jb);
    } else if (out) {
      out[0] = (uint32_t)ja;
      out[a.hit_stride] = (uint32_t)jb;  // (the last one twice: past the list's length)
      out += 2 * (size_t)a.hit_stride;
    }
  };
  fetch(hits);
  for (; hits > 0; hits -= 2) {
    const float4 x0 = xa, x1 = xb, v0 = va, v1 = vb;
    if (hits > 2) fetch(hits - 2);
    p.visit_two(x0, x1, v0, v1, hits > 1);
  }
}

// Codes of PassArgs::hit_n besides a list's length.
enum HitCode : int {
  kHitsDense = -1,  // the particle went to the dense kernel
  kHitsWalk = -2,   // no list: the delta_p passes walk the window again
  kHitsMasks = -3,  // kHitsMasks - k: k chunks with hits (mask, first slot) in place of the list
};

// Chunk k with hits of list slot h.
__device__ __forceinline__ void put_chunk(const PassArgs& a, int h, int k, uint32_t m, uint32_t base) {
  uint32_t* out = a.hits + 2 * (size_t)k * a.hit_stride + h;
  out[0] = m;
  out[a.hit_stride] = base;
}

// Visits the hits of one chunk in order, two at a time.
template <int kKind, class P>
__device__ __forceinline__ void visit_mask(const PassArgs& a, uint32_t m, int base, P& p) {
  while (m) {
    const int ba = __clz(m), ja = base + ba;
    m ^= 0x80000000u >> ba;
    const bool two = m != 0u;
    const int bb = two ? __clz(m) : ba, jb = base + bb;
    if (two) m ^= 0x80000000u >> bb;
    const float4 xa = __ldg(a.X + ja), xb = __ldg(a.X + jb);
    if constexpr (kKind == kXsph)
      p.visit_two(xa, xb, __ldg(a.VR + ja), __ldg(a.VR + jb), two);
    else
      p.visit_two(xa, xb, xa, xb, two);
  }
}

// The chunks (up to 32 candidates from a multiple of four) of run r of the
// window, in order: f(base, groups of four, the candidates that belong to it).
template <class F>
__device__ __forceinline__ void for_chunks(uint2 run, F&& f) {
  const int s = (int)run.x, e = (int)run.y;
  uint32_t valid = 0xffffffffu >> (s & 3);  // drops candidates before s from the first mask
  for (int base = s & ~3; base < e; base += 32) {
    if (e - base < 32) valid &= ~(0xffffffffu >> (e - base));
    f(base, min((e - base + 3) >> 2, 8), valid);
    valid = 0xffffffffu;
  }
}

// Visits the queued hits (n entries) of one particle; returns the code of list
// slot h, which the lambda pass fills: the hits, or where a warp has a particle
// with more than fit its chunks (so that the delta_p pass's warps take one path).
template <int kKind, bool kSecond, class P>
__device__ __forceinline__ int finish_queued(const PassArgs& a, QueueColumn col, int n, int hits, P& p, int h) {
  if (kKind == kLambda && h >= a.hit_stride) {  // no list (the same answer for the warp)
    visit_queued<kKind, kSecond, kSparseThreads>(a, col, hits, p, nullptr);
    return kHitsWalk;
  }
  const bool list = kKind == kLambda && __all_sync(__activemask(), hits <= kHitCap);
  visit_queued<kKind, kSecond, kSparseThreads>(a, col, hits, p, list ? a.hits + h : nullptr);
  if (kKind != kLambda || list) return hits;
  int chunks = 0;
  for (int k = 0; k < n; ++k) {
    const uint2 e = col.run[k * kSparseThreads];
    const uint32_t m = kSecond ? col.second[k * kSparseThreads] : e.x;
    if (m) put_chunk(a, h, chunks++, m, e.y);
  }
  return kHitsMasks - chunks;
}

// The hits of the window whose runs are in the column, visited in order;
// returns the code of list slot h (lambda).  fits: the queue takes the whole
// window (window_runs).  A window of more chunks is one of piled-up particles,
// whose chunks hold many hits each: they are visited chunk by chunk, straight
// from the mask.
template <int kKind, class P>
__device__ __forceinline__ int walk_hits(const PassArgs& a, QueueColumn col, P& p, int h, bool fits) {
  const HitTest test(p.xi, a.c.h2);
  int n = 0, hits = 0;
  for (int r = 0; r < 9; ++r) {
    for_chunks(col.run[(kRunSlot + r) * kSparseThreads], [&](int base, int groups, uint32_t valid) {
      uint32_t m = 0u;
#pragma unroll 2
      for (int g = 0; g < groups; ++g) m = test.four(Four(a.S, a.stride, base + 4 * g), m);
      m = ~m << (32 - 4 * groups) & valid;  // hits, the first candidate in the highest bit
      if (!m) return;
      if (fits) {
        col.run[n * kSparseThreads] = make_uint2(m, (uint32_t)base);
        hits += __popc(m);
      } else {
        if (kKind == kLambda && n < kHitCap / 2 && h < a.hit_stride) put_chunk(a, h, n, m, (uint32_t)base);
        visit_mask<kKind>(a, m, base, p);
      }
      ++n;
    });
  }
  if (fits) return finish_queued<kKind, false>(a, col, n, hits, p, h);
  return kKind == kLambda && n <= kHitCap / 2 && h < a.hit_stride ? kHitsMasks - n : (int)kHitsWalk;
}

// The same walk for two particles of one cell, up to the queue: the masks of
// both (run.x, second); returns the entries and the hits of each.  The caller
// has checked that the window's chunks fit (window_runs).
__device__ __forceinline__ int3 queue_pair(const PassArgs& a, QueueColumn col, float4 x0, float4 x1) {
  const HitTest t0(x0, a.c.h2), t1(x1, a.c.h2);
  int n = 0;
  int3 hits = make_int3(0, 0, 0);
  for (int r = 0; r < 9; ++r) {
    for_chunks(col.run[(kRunSlot + r) * kSparseThreads], [&](int base, int groups, uint32_t valid) {
      uint32_t m0 = 0u, m1 = 0u;
#pragma unroll 2
      for (int g = 0; g < groups; ++g) {
        const Four f(a.S, a.stride, base + 4 * g);
        m0 = t0.four(f, m0);
        m1 = t1.four(f, m1);
      }
      const int sh = 32 - 4 * groups;
      m0 = ~m0 << sh & valid;
      m1 = ~m1 << sh & valid;
      if (m0 | m1) {
        col.run[n * kSparseThreads] = make_uint2(m0, (uint32_t)base);
        col.second[n * kSparseThreads] = m1;
        ++n;
        hits.x += __popc(m0);
        hits.y += __popc(m1);
      }
    });
  }
  hits.z = n;
  return hits;
}

// Visits the first n particles of a hit list in order, kListAhead loads in
// flight (the last batch is filled up with the particle itself, which adds
// nothing).
constexpr int kListAhead = 4;
template <class P>
__device__ __forceinline__ void visit_list(const PassArgs& a, const uint32_t* __restrict__ list, int n, int i, P& p) {
  int j[kListAhead];
#pragma unroll
  for (int u = 0; u < kListAhead; ++u) j[u] = u < n ? (int)__ldg(list + (size_t)u * a.hit_stride) : i;
  for (int k = 0; k < n; k += kListAhead) {
    float4 x[kListAhead];
#pragma unroll
    for (int u = 0; u < kListAhead; ++u) x[u] = __ldg(a.X + j[u]);
    list += (size_t)kListAhead * a.hit_stride;
#pragma unroll
    for (int u = 0; u < kListAhead; ++u)
      j[u] = k + kListAhead + u < n ? (int)__ldg(list + (size_t)u * a.hit_stride) : i;
#pragma unroll
    for (int u = 0; u < kListAhead; u += 2) p.visit_two(x[u], x[u + 1], x[u], x[u + 1], true);
  }
}

// Visits the hits of the n chunks that took the list's place, the next chunk's
// load issued one ahead.
template <int kKind, class P>
__device__ __forceinline__ void visit_chunks(const PassArgs& a, const uint32_t* __restrict__ list, int n, P& p) {
  if (n == 0) return;
  uint32_t m = __ldg(list), base = __ldg(list + a.hit_stride);
  for (int k = 1; k <= n; ++k) {
    list += 2 * (size_t)a.hit_stride;
    const uint32_t mn = k < n ? __ldg(list) : 0u, bn = k < n ? __ldg(list + a.hit_stride) : 0u;
    visit_mask<kKind>(a, m, (int)base, p);
    m = mn;
    base = bn;
  }
}

// Whether walk_hits and the hit lists hold for a particle at xi: keps2 a normal
// number (a pair below it has no gradient; rsqrt_normal), xi finite.
__device__ __forceinline__ bool fast_hits(const PassArgs& a, float4 xi) {
  return a.c.keps2 >= kNormalMin && isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z);
}

// The 9 column runs of the window of cell q into the column; returns the
// candidates they hold.  Every load is issued before the first is used.
// fits: the chunks of any prefix of the runs fit the queue entries that are
// free by then.
__device__ __forceinline__ int window_runs(const SceneGeom& g, const uint32_t* __restrict__ cs, int n, int3 q,
                                           QueueColumn col, bool& fits) {
  const int zlo = max(q.z - 1, 0), zhi = min(q.z + 1, g.dims[2] - 1);
  uint32_t s[9], e[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int x = q.x + r / 3 - 1, y = q.y + r % 3 - 1;
    const bool in = x >= 0 && x < g.dims[0] && y >= 0 && y < g.dims[1];
    const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
    s[r] = in ? __ldg(cs + base + zlo) : 0u;
    e[r] = in ? __ldg(cs + base + zhi + 1) : 0u;
  }
  int total = 0, chunks = 0;
  fits = true;
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int end = max(min((int)e[r], n), (int)s[r]);  // as column_run
    col.run[(kRunSlot + r) * kSparseThreads] = make_uint2(s[r], (uint32_t)end);
    total += end - (int)s[r];
    chunks += end > (int)s[r] ? (end - (int)(s[r] & ~3u) + 31) >> 5 : 0;
    fits = fits && chunks <= kRunSlot + r + 1;
  }
  return total;
}

// Appends the first `count` (0, 1 or 2) of slots t, t + 1 of every lane to the
// dense list, in slot order (one atomic per warp; every lane of the warp calls
// it).
__device__ __forceinline__ void append_dense(const PassArgs& a, int count, int t) {
  const unsigned one = __ballot_sync(kFull, count > 0), two = __ballot_sync(kFull, count > 1);
  if (!one) return;
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  uint32_t base = 0u;
  if (lane == 0) base = atomicAdd(&a.flags[a.counter], (uint32_t)(__popc(one) + __popc(two)));
  base = __shfl_sync(kFull, base, 0) + (uint32_t)(__popc(one & lt) + __popc(two & lt));
  if (count > 0) a.dense[base] = (uint32_t)t;
  if (count > 1) a.dense[base + 1u] = (uint32_t)t + 1u;
}

// A particle whose window of `entries` entries the sparse kernel walks, on its
// own: group by group (grouped), every candidate (exact), or its hits; h: its
// hit list's slot.
template <int kKind>
__device__ __forceinline__ void sparse_one(const PassArgs& a, const SceneGeom& g, int3 q, QueueColumn col, int h,
                                           int i, float4 xi, bool exact, bool grouped, int entries, bool fits) {
  typename PassOf<kKind>::type p(a, g, xi, i, exact);
  int code = kHitsWalk;
  if (grouped || exact || !fast_hits(a, xi)) {
    HitQueue hq(nullptr, nullptr, kSparseThreads, 1);
    const FromGlobal src{a.X};
    if (grouped)
      visit_window_grouped(g, a, q, src, p, 0, entries, hq);
    else if (exact)
      visit_window(g, a.cs, a.n, q, src, p);  // non-neighbours matter: visit every candidate
    else
      visit_window_masked(g, a.cs, a.n, q, src, p, hq);
  } else {
    code = walk_hits<kKind>(a, col, p, h, fits);
  }
  p.finish(a);
  if (kKind == kLambda) a.hit_n[h] = code;
}

// PBF_SPARSE_MIN_BLOCKS (a build-time tuning macro): resident blocks per SM the
// compiler must allow for, which caps the sparse kernels' registers.
#ifdef PBF_SPARSE_MIN_BLOCKS
#define PBF_SPARSE_BOUNDS __launch_bounds__(kSparseThreads, PBF_SPARSE_MIN_BLOCKS)
#else
#define PBF_SPARSE_BOUNDS __launch_bounds__(kSparseThreads)
#endif

// One thread slot of the pass's list (or of all particles) per thread; the
// grid covers every slot, blocks past the list's end return at once.  The
// delta_p passes, and the others where the particles are not paired.
//
// The delta_p passes take the hits the lambda pass listed: each list entry
// costs one coalesced load and one gathered one (position and lambda), kept
// kListAhead ahead, and two entries share the packed arithmetic.  Bound by the
// gathers (L1 data path 70% busy: 32 lanes' neighbours lie in ~10 lines).
// 1,048,576 particles at rest density: 167 -> 77 us a pass (saved masks, whose
// bits a warp visits chunk by chunk, before).
template <int kKind>
__global__ void PBF_SPARSE_BOUNDS k_sparse(PassArgs a) {
  using P = typename PassOf<kKind>::type;
  constexpr bool kDp = kKind == kDeltaP || kKind == kDeltaPFinal;
  __shared__ uint2 queue[kQueueSlots * kSparseThreads];
  const int count = work_count(a);
  const bool apart = a.paired && a.flags[kGroupCount] != 0u;  // pair_slots: a particle on every even slot
  if ((int)(blockIdx.x * kSparseThreads << (apart ? 1 : 0)) >= count) return;  // uniform over the block
  const QueueColumn col{queue + threadIdx.x, nullptr};
  // h: the thread's hit list.  Paired, the lambda pass's warp w lists the first
  // particles of its 32 pairs at 64 w + lane and the second ones at 64 w + 32 +
  // lane, so that its stores and these loads take consecutive words; apart, pair
  // h's particle at h.
  const int h = blockIdx.x * kSparseThreads + threadIdx.x;
  const int t = apart ? 2 * h : (a.paired ? (h & ~63) + 2 * (h & 31) + (h >> 5 & 1) : h);
  const int i = t < count ? work_particle(a, t) : -1;
  const bool valid = i >= 0;
  const float4 xi = valid ? a.X[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const SceneGeom g = geom_of(a.c, a.G, valid ? i : 0);
  // the delta_p passes take the lambda pass's routing and list where it left one
  const int code = kDp && valid ? a.hit_n[h] : kHitsWalk;
  const bool listed = kDp && (code >= 0 || code <= kHitsMasks);
  const bool walk = valid && !listed && code != kHitsDense;
  int3 q = make_int3(0, 0, 0);
  int entries = 0;
  bool grouped = false, fits = false;
  if (walk) {
    q = cell_of(a.c, g, xi);
    entries = window_runs(g, a.cs, a.n, q, col, fits);
    // a window over dense_window candidates that its grouped cells bring back
    // under it is walked here, group by group
    grouped = entries > a.c.dense_window && a.c.keps2 > 0.f && a.flags[kGroupCount] != 0u;
    if (grouped) entries = window_total_grouped(g, a, q);
  }
  // a window over dense_window entries goes to the dense kernel, particle by
  // particle: which kernel sums a particle's window depends on its own window
  // only, so results do not depend on the list's order or on the particle's
  // warp-mates
  const bool go_dense = valid && (walk ? entries > a.c.dense_window : code == kHitsDense);
  append_dense(a, go_dense ? 1 : 0, t);
  // one path per warp (its lanes' windows mostly agree)
  fits = __all_sync(kFull, fits || !walk || go_dense || grouped);
  if (!valid) return;
  if (go_dense) {
    // a window with groups may count them again after the sums of lambda
    if (kKind == kLambda) a.hit_n[h] = grouped ? kHitsWalk : kHitsDense;
    return;
  }
  if (kDp && !walk && a.flags[kFlagLambdaNonFinite]) q = cell_of(a.c, g, xi);  // for exact_path
  const bool exact = exact_path(kKind, a, g, q, i);
  if (kDp && !walk && !exact) {
    P p(a, g, xi, i, exact);
    if (code >= 0)
      visit_list(a, a.hits + h, code, i, p);
    else
      visit_chunks<kKind>(a, a.hits + h, kHitsMasks - code, p);
    p.finish(a);
  } else {
    sparse_one<kKind>(a, g, q, col, h, i, xi, exact, grouped, entries, fits);
  }
}

// The lambda and xsph passes over paired buckets: two particles of one cell
// per thread.  They share the window, so the candidates' loads and the walk
// serve both; the hits are then visited one particle after the other.
//
// Bound by the L1 data path and instruction issue: a test reads 12 bytes per
// lane whatever the lanes share (L1 returns 128 bytes a cycle), 800 cycles for
// 32 particles when every thread tested for one.  1,048,576 particles at rest
// density: lambda 226 -> 145 us, xsph 260 -> 212 us; one particle per thread
// with the same queue and packed arithmetic 169 and 215.  Eight blocks (64
// registers) beat seven (no spills) and nine by 1 and 4% of the step.
template <int kKind>
__global__ void __launch_bounds__(kSparseThreads, 8) k_sparse_pair(PassArgs a) {
  using P = typename PassOf<kKind>::type;
  __shared__ uint2 queue[kQueueSlots * kSparseThreads];
  __shared__ uint32_t second[kQueueSlots * kSparseThreads];
  const int count = work_count(a);  // even
  if ((int)(2 * blockIdx.x * kSparseThreads) >= count) return;  // uniform over the block
  const QueueColumn col{queue + threadIdx.x, second + threadIdx.x};
  const int pair = blockIdx.x * kSparseThreads + threadIdx.x;
  // hit list of the first; the second's is h + 32 (see k_sparse)
  const int h = a.flags[kGroupCount] != 0u ? pair : 2 * (pair & ~31) + (pair & 31);
  const bool valid = 2 * pair < count;
  const int2 i = valid ? __ldg(reinterpret_cast<const int2*>(a.list) + pair) : make_int2(-1, -1);
  const bool two = i.y >= 0;
  const float4 x0 = valid ? a.X[i.x] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 x1 = two ? a.X[i.y] : x0;
  const SceneGeom g = geom_of(a.c, a.G, valid ? i.x : 0);
  const int3 q = cell_of(a.c, g, x0);  // x1's too
  int entries = 0;
  bool grouped = false, fits = false;
  if (valid) {
    entries = window_runs(g, a.cs, a.n, q, col, fits);
    grouped = entries > a.c.dense_window && a.c.keps2 > 0.f && a.flags[kGroupCount] != 0u;
    if (grouped) entries = window_total_grouped(g, a, q);
  }
  const bool go_dense = valid && entries > a.c.dense_window;  // as in k_sparse
  append_dense(a, go_dense ? (two ? 2 : 1) : 0, 2 * pair);
  fits = __all_sync(kFull, fits || !valid || go_dense || grouped);
  if (!valid) return;
  if (go_dense) {
    if (kKind == kLambda) {
      a.hit_n[h] = grouped ? kHitsWalk : kHitsDense;
      if (two) a.hit_n[h + 32] = a.hit_n[h];
    }
    return;
  }
  bool plain = true;  // xsph: k_xsph_poison looks for what poisons the sums (see there)
  if (kKind == kXsph && a.flags[kFlagXsphExact] != 0u) {
    if (a.flags[kGroupCount] != 0u)  // (one particle per pair then)
      plain = !exact_path(kKind, a, g, q, i.x) && (!two || !exact_path(kKind, a, g, q, i.y));
    else
      plain = tame(a.VR[i.x]) && (!two || tame(a.VR[i.y]));
  }
  if (!grouped && plain && fits && fast_hits(a, x0) && fast_hits(a, x1)) {
    const int3 hits = queue_pair(a, col, x0, x1);
    {
      P p(a, g, x0, i.x, false);
      const int code = finish_queued<kKind, false>(a, col, hits.z, hits.x, p, h);
      p.finish(a);
      if (kKind == kLambda) a.hit_n[h] = code;
    }
    if (two) {
      P p(a, g, x1, i.y, false);
      const int code = finish_queued<kKind, true>(a, col, hits.z, hits.y, p, h + 32);
      p.finish(a);
      if (kKind == kLambda) a.hit_n[h + 32] = code;
    }
    return;
  }
  for (int u = 0; u < (two ? 2 : 1); ++u) {
    bool f;
    if (u) window_runs(g, a.cs, a.n, q, col, f);  // the first walk's queue has taken their place
    const int k = u ? i.y : i.x;
    sparse_one<kKind>(a, g, q, col, h + 32 * u, k, u ? x1 : x0, exact_path(kKind, a, g, q, k), grouped, entries, fits);
  }
}

// The exact path of the xsph pass over pairs, for the particles whose neighbours
// k_sparse_pair took as ever: the candidates beyond them that poison the sum of a
// tame particle lie in cells that hold a particle with such a density or
// velocity now (k_xsph_mark; kCellRhoNotPositive has gathered those of every
// iteration), a few of a window's 27.  Nothing to do, but for two launches (3 us
// each), in a step without any.  The exact walk, which visits every candidate of
// the window, held up its warp's other lanes: the pass in an ensemble of
// 4,714,514 particles (4,303 of them not finite) 1,933 -> 735 us and 326 for
// these two; the same code in k_sparse_pair spilled and cost a step without such
// particles 50 us; a warp per particle, a lane per cell, took 1,048 us.  Steps
// with grouped cells keep the walk (1,048,576 clustered particles: the pass 178 us,
// 204 this way).
__global__ void __launch_bounds__(256) k_xsph_mark(PassArgs a) {
  if (a.flags[kFlagXsphExact] == 0u || a.flags[kGroupCount] != 0u) return;
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= a.n) return;
  const float4 vr = a.VR[i];
  if (vr.w > 0.f && isfinite(vr.w) && isfinite(vr.x) && isfinite(vr.y) && isfinite(vr.z)) return;
  uint32_t* f = a.cell_flags + a.skeys[i];
  if (!(*reinterpret_cast<volatile uint32_t*>(f) & kCellPoison)) atomicOr(f, (uint32_t)kCellPoison);
}

__global__ void __launch_bounds__(256) k_xsph_poison(PassArgs a) {
  if (a.flags[kFlagXsphExact] == 0u || a.flags[kGroupCount] != 0u) return;
  const int pair = blockIdx.x * 256 + threadIdx.x;
  if (2 * pair >= work_count(a)) return;
  const int2 i = __ldg(reinterpret_cast<const int2*>(a.list) + pair);
  const bool two = i.y >= 0;
  const float4 x0 = a.X[i.x], x1 = two ? a.X[i.y] : x0;
  const SceneGeom g = geom_of(a.c, a.G, i.x);
  const int3 q = cell_of(a.c, g, x0);  // x1's too
  uint32_t cells = 0u;
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const int x = q.x + k / 9 - 1, y = q.y + k / 3 % 3 - 1, z = q.z + k % 3 - 1;
    const bool in = (unsigned)x < (unsigned)g.dims[0] && (unsigned)y < (unsigned)g.dims[1] &&
                    (unsigned)z < (unsigned)g.dims[2];
    if (in && (a.cell_flags[cell_index(g, x, y, z)] & kCellPoison)) cells |= 1u << k;
  }
  if (cells == 0u || !fast_hits(a, x0) || !fast_hits(a, x1)) return;
  XsphPass p0(a, g, x0, i.x, true), p1(a, g, x1, two ? i.y : i.x, true);
  if (!tame(a.VR[i.x]) || (two && !tame(a.VR[i.y]))) return;  // (walked candidate by candidate)
  for (; cells; cells &= cells - 1u) {
    const int k = __ffs(cells) - 1;
    const int cell = cell_index(g, q.x + k / 9 - 1, q.y + k / 3 % 3 - 1, q.z + k % 3 - 1);
    const int s = (int)__ldg(a.cs + cell), e = min((int)__ldg(a.cs + cell + 1), a.n);
    if (e - s > a.c.dense_window) return;  // the window is the dense kernel's, or walked with its groups
    for (int j = s; j < e; ++j) {
      const float4 xj = __ldg(a.X + j), vj = __ldg(a.VR + j);
      p0.miss_beyond(xj, vj);
      p1.miss_beyond(xj, vj);
    }
  }
  const float qnan = __int_as_float(0x7fffffff);
  for (int u = 0; u < (two ? 2 : 1); ++u) {
    const XsphPass& p = u ? p1 : p0;
    if (p.px) a.NV[p.i].x = qnan;
    if (p.py) a.NV[p.i].y = qnan;
    if (p.pz) a.NV[p.i].z = qnan;
  }
}

// PBF_DENSE_BLOCKS_PER_SM (a build-time tuning macro, pbf_internal.cuh): the
// dense kernel's resident blocks per SM, which its grid is sized for and its
// registers are capped to.
#define PBF_DENSE_BOUNDS __launch_bounds__(kDenseThreads, PBF_DENSE_BLOCKS_PER_SM)

// kStage: the variant that stages each item's column runs (launched when
// stage_dense > 0); the other carries no staging code.
// A part of a window without grouped cells, entries [lo, hi) in visiting order,
// for a particle that walk_hits would take: the sparse kernel's tests and packed
// visits.  runs: the window's, 32 apart; q: this thread's queue column.  Where
// saved is not null the lambda pass leaves the part's chunks with hits there (up
// to cap of them: mask, first slot; a zero mask ends them, and a slot of ~0 there
// says that they did not fit).
constexpr int kPartQueue = 4;
template <int kKind, class P>
__device__ __forceinline__ void visit_part(const PassArgs& a, const uint2* runs, int lo, int hi, P& p, QueueColumn q,
                                           uint32_t* saved, int cap) {
  const HitTest test(p.xi, a.c.h2);
  int v0 = 0, chunks = 0, n = 0, hits = 0;
  for (int r = 0; r < 9; ++r) {
    const uint2 run = runs[32 * r];
    const int len = (int)(run.y - run.x);
    const int from = max(lo - v0, 0), to = min(hi - v0, len);
    v0 += len;
    if (from >= to) continue;
    for_chunks(make_uint2(run.x + from, run.x + to), [&](int base, int groups, uint32_t valid) {
      uint32_t m = 0u;
#pragma unroll 4
      for (int g = 0; g < groups; ++g) m = test.four(Four(a.S, a.stride, base + 4 * g), m);
      m = ~m << (32 - 4 * groups) & valid;
      if (!m) return;
      if (n == kPartQueue) {
        visit_queued<kKind, false, kDenseThreads>(a, q, hits, p, nullptr);
        n = hits = 0;
      }
      q.run[n * kDenseThreads] = make_uint2(m, (uint32_t)base);
      ++n;
      hits += __popc(m);
      if (saved && chunks < cap) saved[2 * chunks] = m, saved[2 * chunks + 1] = (uint32_t)base;
      ++chunks;
    });
  }
  visit_queued<kKind, false, kDenseThreads>(a, q, hits, p, nullptr);
  if (saved && chunks != cap) {
    const int end = chunks > cap ? 0 : chunks;
    saved[2 * end] = 0u, saved[2 * end + 1] = chunks > cap ? ~0u : 0u;
  }
}

// The first entry of what the lambda pass saved, and whether it says that the
// part's hits are there (not where they did not fit).
__device__ __forceinline__ uint2 saved_entry(const uint32_t* saved, int k) {
  return __ldg(reinterpret_cast<const uint2*>(saved) + k);
}
__device__ __forceinline__ bool saved_fits(uint2 first) { return first.x != 0u || first.y == 0u; }

// The same hits from what the lambda pass saved (saved_fits).
template <int kKind, class P>
__device__ __forceinline__ void visit_saved(const PassArgs& a, P& p, QueueColumn q, const uint32_t* saved, uint2 first,
                                            int cap) {
  int n = 0, hits = 0;
  uint2 e = first;
  for (int k = 0; k < cap; ++k) {
    if (k) e = saved_entry(saved, k);
    if (e.x == 0u) break;
    if (n == kPartQueue) {
      visit_queued<kKind, false, kDenseThreads>(a, q, hits, p, nullptr);
      n = hits = 0;
    }
    q.run[n * kDenseThreads] = e;
    ++n;
    hits += __popc(e.x);
  }
  visit_queued<kKind, false, kDenseThreads>(a, q, hits, p, nullptr);
}

// Steps of few particles are bound by the latency of a pass's chain of loads,
// not by its work, so the chain is kept short: a block's first batch is its
// own index, the runs of the batch's windows are loaded by all its warps at once
// and shared, a part's tests have twelve 16-byte loads in flight, and where every
// particle is dense the delta_p passes take the hits the lambda pass saved.
// 1,728 particles: lambda 13.1 -> 9.0 us, delta_p 15.7 -> 7.6;
// 65,231: 36 -> 37 and 43 -> 29.
template <int kKind, bool kStage>
__global__ void PBF_DENSE_BOUNDS k_dense(PassArgs a) {
  using P = typename PassOf<kKind>::type;
  constexpr bool kDp = kKind == kDeltaP || kKind == kDeltaPFinal;
  __shared__ float part[kDenseWarps][kMaxFields][32];
  __shared__ StageState st;
  __shared__ uint2 window[kStage ? 1 : kDenseWarps][kStage ? 1 : 9][32];
  __shared__ uint2 queue[kStage ? 1 : kPartQueue * kDenseThreads];
  // dynamic shared memory: the hit queue (a.c.queue_dense chunks per thread),
  // then the stage (a.c.stage_dense slots, kStage only)
  extern __shared__ __align__(16) float4 dyn_smem[];
  uint32_t* q_mask = reinterpret_cast<uint32_t*>(dyn_smem);
  int* q_base = reinterpret_cast<int*>(q_mask + a.c.queue_dense * kDenseThreads);
  float4* stage = dyn_smem + a.c.queue_dense * kDenseThreads / 2;
  static_assert(P::kFields <= kMaxFields, "partial-sum fields");
  HitQueue hq(q_mask + threadIdx.x, q_base + threadIdx.x, kDenseThreads, a.c.queue_dense);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cap = kStage ? a.c.stage_dense : 0;
  if (kStage && threadIdx.x == 0 && cap > 0) stage_init(st);
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // their pass has finished
    a.flags[a.next_counter] = 0u;
    a.flags[a.next_item_counter] = 0u;
  }
  // the slots the sparse kernel listed, or all of them, 32 per item
  const int work = work_count(a);
  const uint32_t listed = a.flags[kStepFailed] ? 0u : (a.dense_all ? (uint32_t)work : a.flags[a.counter]);
  const uint32_t count = (listed + 31) / 32;
  // kSplit warps share an item (each walks one contiguous part of every
  // lane's window); the block runs kDenseWarps / kSplit items at a time.  The
  // staged variant gives each item the whole block.
  const int split = kStage ? kDenseWarps : a.c.dense_split;  // 1, 2, 4 or 8
  const int split_log2 = 31 - __clz(split);
  const int slots = kDenseWarps >> split_log2;
  const int slot = warp >> split_log2, sub = warp & (split - 1);
  // no grouped cell this step: windows are walked as 9 column runs (the same
  // candidates in the same order as cell by cell, with fewer table reads)
  const bool groups = a.c.keps2 > 0.f && a.flags[kGroupCount] != 0u;
  const bool flat = !kStage && !groups && !a.c.dense_interleave;
  // a part's share of a particle's 64 words in a.hits (the sparse kernel's lists
  // are not in use then)
  const int words = kHitCap >> split_log2;
  const bool saves = flat && a.dense_all && a.hits != nullptr;
  // a block's first batches are its index's; then batches are handed out one
  // block-load at a time by a counter, so a block that drew light batches takes
  // more (batches cost from a few hundred to many thousand candidates); which
  // block computes a batch changes nothing
  __shared__ uint32_t s_first;
  uint32_t phase = 0u;
  const uint32_t own = gridDim.x * (uint32_t)slots;
  for (bool once = true;; once = false) {
    uint32_t first = blockIdx.x * (uint32_t)slots;
    if (!once) {
      if (own >= count) break;  // uniform over the grid: every batch was some block's own
      if (threadIdx.x == 0) s_first = own + atomicAdd(&a.flags[a.item_counter], (uint32_t)slots);
      __syncthreads();  // also: every thread has read the previous s_first
      first = s_first;
    }
    if (first >= count) break;  // uniform over the block
    const uint32_t item = first + (uint32_t)slot;
    const uint32_t e = item * 32 + lane;
    const bool valid = item < count && e < listed;
    const int t = valid ? (int)(a.dense_all ? e : a.dense[e]) : 0;
    const int i = valid ? work_particle(a, t) : 0;
    const float4 xi = valid ? a.X[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneGeom g = geom_of(a.c, a.G, valid ? i : 0);
    const int3 q = cell_of(a.c, g, xi);
    const bool exact = valid && exact_path(kKind, a, g, q, i);
    // the item's windows staged in shared memory: every warp holds the same
    // 32 particles, so warp 0's vote is the block's (block-uniform branch)
    bool staged = false;
    if (kStage && cap > 0) {
      if (warp == 0) stage_vote(st, 0, valid, g, q, i);
      __syncthreads();  // also: the previous item's reads of the stage are done
      if (threadIdx.x == 0) stage_issue(st, 1, a, stage, cap);
      __syncthreads();
      staged = stage_wait(st, a, phase);
    }
    uint32_t* saved = saves ? a.hits + (size_t)t * kHitCap + sub * words : nullptr;
    const bool fast = flat && !exact && fast_hits(a, xi);
    if (flat) {  // the windows' runs, each of the item's warps its share of the nine
      if (valid)
        for (int r = sub; r < 9; r += split) {
          int s0 = 0, e0 = 0;
          const int x = q.x + r / 3 - 1, y = q.y + r % 3 - 1;
          if (x >= 0 && x < g.dims[0] && y >= 0 && y < g.dims[1]) column_run(g, a.cs, a.n, x, y, q.z, s0, e0);
          window[kStage ? 0 : slot][kStage ? 0 : r][lane] = make_uint2((uint32_t)s0, (uint32_t)e0);
        }
      __syncthreads();
    }
    if (valid) {
      P p(a, g, xi, i, exact);
      const QueueColumn col{queue + (kStage ? 0 : threadIdx.x), nullptr};
      const bool look = kDp && fast && saves;
      const uint2 entry = look ? saved_entry(saved, 0) : make_uint2(0u, ~0u);
      if (look && saved_fits(entry)) {  // the lambda pass's hits
        visit_saved<kKind>(a, p, col, saved, entry, words / 2);
      } else {
        int total = 0;
        if (flat) {
          for (int r = 0; r < 9; ++r) {
            const uint2 run = window[kStage ? 0 : slot][kStage ? 0 : r][lane];
            total += (int)(run.y - run.x);
          }
        } else {
          total = groups ? window_total_grouped(g, a, q) : window_total(g, a.cs, a.n, q);
        }
        const int lo = (int)(((long long)total * sub) >> split_log2);
        const int hi = (int)(((long long)total * (sub + 1)) >> split_log2);
        // a staged window holds no grouped cell: its runs are walked as runs;
        // dense_interleave: the warps take every split-th chunk instead of
        // one contiguous part (windows without grouped cells)
        if (kStage && staged) {
          if (a.c.dense_interleave)
            visit_window_strided(g, a.cs, a.n, q, FromStage{stage, st.D}, p, sub, split, hq);
          else
            visit_window_chunk(g, a.cs, a.n, q, FromStage{stage, st.D}, p, lo, hi, hq);
        } else if (groups) {
          visit_window_grouped(g, a, q, FromGlobal{a.X}, p, lo, hi, hq);
        } else if (a.c.dense_interleave) {
          visit_window_strided(g, a.cs, a.n, q, FromGlobal{a.X}, p, sub, split, hq);
        } else if (fast) {
          visit_part<kKind>(a, &window[kStage ? 0 : slot][0][lane], lo, hi, p, col,
                            kKind == kLambda ? saved : nullptr, words / 2);
        } else {
          visit_window_chunk(g, a.cs, a.n, q, FromGlobal{a.X}, p, lo, hi, hq);
        }
      }
      p.store(&part[warp][0][lane], 32);
    }
    __syncthreads();
    if (sub == 0 && valid) {
      P p(a, g, xi, i, exact);
      for (int k = 0; k < split; ++k) p.add(&part[slot * split + k][0][lane], 32);
      p.finish(a);
    }
    __syncthreads();
  }
  if (kStage && cap > 0) stage_drain(st, phase);
}

// Also registers every cell holding >= kGroupCell particles (its first
// particle takes a group slot).  flags and cell_flags start at zero.
__global__ void __launch_bounds__(256)
k_reorder(const uint32_t* __restrict__ perm, const float4* __restrict__ pos,
          const float4* __restrict__ vel, const uint32_t* __restrict__ iid, int n, StepConsts c,
          float4* __restrict__ xs, float4* __restrict__ xa, float* __restrict__ sa, int stride,
          uint32_t* __restrict__ iid_s, uint32_t* __restrict__ flags, const uint32_t* __restrict__ skeys,
          const uint32_t* __restrict__ cs, uint32_t* __restrict__ cell_flags, int* __restrict__ grp_cell,
          int* __restrict__ grp_off, int* __restrict__ grp_item_off, int* __restrict__ grp_item_slot, int chunk) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  if (k == 0) flags[kDirtyWord] = 0u;  // the grid's clear has seen to it
  const uint32_t key = skeys[k];
  const uint32_t pop = cs[key + 1] - cs[key];
  if ((uint32_t)k == cs[key] && pop >= (uint32_t)kGroupCell) {
    // one slot per such cell (< n / kGroupCell of them) and `pop` pool entries
    // (the pool holds n: the cells' populations sum to <= n)
    const uint32_t slot = atomicAdd(&flags[kGroupCount], 1u);
    grp_cell[slot] = (int)key;
    grp_off[slot] = (int)atomicAdd(&flags[kGroupPool], pop);
    // work items of `chunk` particles (< n / chunk + slots of them)
    const int items = (int)((pop + chunk - 1) / chunk);
    const int i0 = (int)atomicAdd(&flags[kGroupItems], (uint32_t)items);
    grp_item_off[slot] = i0;
    for (int t = 0; t < items; ++t) grp_item_slot[i0 + t] = (int)slot;
    atomicOr(&cell_flags[key], (slot + 1u) << kCellSlotShift);
  }
  const uint32_t p = min(perm[k], (uint32_t)(n - 1));  // a permutation of [0, n): the min never binds
  const float4 x = pos[p];
  const float4 v = vel[p];
  const float vx = fmaf(c.dt, c.g[0], v.x), vy = fmaf(c.dt, c.g[1], v.y),
              vz = fmaf(c.dt, c.g[2], v.z);
  xs[k] = x;
  const float4 xp = make_float4(fmaf(c.dt, vx, x.x), fmaf(c.dt, vy, x.y), fmaf(c.dt, vz, x.z), x.w);
  xa[k] = xp;
  put_components(sa, stride, k, xp);
  iid_s[k] = iid[p];
}

// ---- group tables ----------------------------------------------------------------------

enum GroupsWhat { kGroupsPos = 0, kGroupsLambda = 1, kGroupsXsph = 2 };

constexpr int kGroupThreads = 1024;
constexpr int kGroupWarps = kGroupThreads / 32;
constexpr int kGroupList = 4096;  // groups ranked in shared memory; more: an ordered scan

struct GroupArgs {
  const float4* X;        // positions of the pass
  const float4* V;        // xsph: velocities
  const float* rho;       // xsph: densities
  const float* lambda;    // delta_p: lambda
  const uint32_t* cs;
  const uint32_t* flags;  // flags[kGroupCount]: slots, flags[kGroupItems]: work items
  int n;
  int np;                 // pool entries
  int chunk;              // particles of a work item
  const int* cell;
  const int* off;
  const int* item_off;    // first work item of each slot
  const int* item_slot;   // slot of each work item
  int* done;              // per slot: work items finished (last-block-done; back to 0 after use)
  int* ng;
  int* rep;
  int* cnt;
  float4* pos;
  float4* sum;
  float4* aux;
  int* id;                // hash entry of each particle of a grouped cell
  int* hash;              // owner (k + 1), count, first (0x7fffffff - k), rank: 2 np each; 0 = empty
  int* list;              // pool: entries claimed per slot
  int* list_n;            // per slot: entries claimed
  unsigned* gmax;
  unsigned long long* acc;
  int* zero;              // per slot: every deviation is zero
};

// The key of particle j: the values that enter a pair term non-linearly.
template <int kWhat>
struct GroupKey {
  static constexpr int kWords = kWhat == kGroupsXsph ? 4 : 3;
  uint32_t w[kWords];
  GroupKey() = default;
  __device__ __forceinline__ GroupKey(const GroupArgs& a, int j) {
    const float4 x = a.X[j];
    w[0] = __float_as_uint(x.x), w[1] = __float_as_uint(x.y), w[2] = __float_as_uint(x.z);
    if constexpr (kWhat == kGroupsXsph) w[3] = __float_as_uint(a.rho[j]);
  }
  __device__ __forceinline__ bool operator==(const GroupKey& o) const {
    bool eq = true;
    for (int k = 0; k < kWords; ++k) eq &= w[k] == o.w[k];
    return eq;
  }
  __device__ __forceinline__ uint32_t hash() const {
    uint32_t h = 0x9e3779b9u;
    for (int k = 0; k < kWords; ++k) {
      h ^= w[k] + 0x7f4a7c15u + (h << 6) + (h >> 2);
      h *= 0x85ebca6bu;
    }
    return h ^ (h >> 15);
  }
};

// x - x_rep, and 0 where the two are the same bits (so a group whose members
// share one non-finite value keeps it).
__device__ __forceinline__ float dev_from(float x, float xr) {
  return __float_as_uint(x) == __float_as_uint(xr) ? 0.f : x - xr;
}

// Exclusive prefix of `flag` over the block in thread order; `total` gets the sum.
__device__ __forceinline__ int block_scan(int flag, int* sh, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned ball = __ballot_sync(0xffffffffu, flag);
  const int in_warp = __popc(ball & ((1u << lane) - 1u));
  __syncthreads();
  if (lane == 0) sh[warp] = __popc(ball);
  __syncthreads();
  if (warp == 0) {
    const int v = lane < kGroupWarps ? sh[lane] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < kGroupWarps) sh[32 + lane] = x - v;  // exclusive
    if (lane == kGroupWarps - 1) sh[64] = x;
  }
  __syncthreads();
  total = sh[64];
  return sh[32 + warp] + in_warp;
}

// Exclusive prefix of `v` over the block in thread order; `total` gets the sum.
__device__ __forceinline__ int block_scan_value(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int w = lane < kGroupWarps ? sh[lane] : 0;
    int y = w;
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    if (lane < kGroupWarps) sh[32 + lane] = y - w;  // exclusive
    if (lane == kGroupWarps - 1) sh[64] = y;
  }
  __syncthreads();
  total = sh[64];
  return sh[32 + warp] + x - v;
}

// A grouped cell's particles in work items of a.chunk; a kernel takes
// items grid-stride and the block that finishes a slot's last item (counted
// in done[slot], made visible by a fence) runs the slot's finishing step and
// sets the counter back to 0.
struct Item {
  int slot, b, m, k0, k1, t0;
};

__device__ __forceinline__ Item item_of(const GroupArgs& a, int item) {
  Item it;
  it.slot = a.item_slot[item];
  const int cell = a.cell[it.slot];
  it.b = (int)a.cs[cell];
  it.m = max(min((int)a.cs[cell + 1], a.n) - it.b, 0);
  it.k0 = (item - a.item_off[it.slot]) * a.chunk;
  it.k1 = min(it.k0 + a.chunk, it.m);
  it.t0 = a.off[it.slot];
  return it;
}

// After a block's share of an item: whether it finished the slot's last item.
__device__ __forceinline__ bool last_item(const GroupArgs& a, const Item& it, int* s_last) {
  __threadfence();  // this block's writes, before the count that may let another block read them
  __syncthreads();
  if (threadIdx.x == 0) {
    const int items = (it.m + a.chunk - 1) / a.chunk;
    *s_last = atomicAdd(&a.done[it.slot], 1) == items - 1;
  }
  __syncthreads();
  if (*s_last) __threadfence();
  return *s_last;
}

// Inserts the item's particles into the slot's hash table (2 entries per
// particle of the cell, so every key finds an entry; integer atomics only),
// kUnroll probe chains per thread in flight.  The block that finishes the
// slot numbers the groups in order of their first particle (by counting in
// shared memory, or for over kGroupList groups by an ordered block scan),
// writes rep, cnt, pos (and for xsph aux = the first particle's velocity and
// sum.w = its density), h_rank, ng, and clears the claimed entries.
template <int kWhat>
__device__ __forceinline__ void group_insert(const GroupArgs& a) {
  __shared__ int sh[80];
  __shared__ int s_last;
  __shared__ int s_buf[2 * kGroupList];
  const int items = (int)a.flags[kGroupItems];
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const Item it = item_of(a, item);
    const int H = 2 * it.m;
    int* h_owner = a.hash + 2 * it.t0;
    int* h_cnt = h_owner + 2 * a.np;
    int* h_first = h_owner + 4 * a.np;
    int* h_rank = h_owner + 6 * a.np;
    int* list = a.list + it.t0;
    constexpr int kUnroll = 4;
    for (int k0 = it.k0 + threadIdx.x; k0 < it.k1; k0 += kUnroll * kGroupThreads) {
      int found[kUnroll];
      GroupKey<kWhat> key[kUnroll];
      int h[kUnroll], o[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = min(k0 + u * kGroupThreads, it.k1 - 1);
        key[u] = GroupKey<kWhat>(a, it.b + k);
        h[u] = (int)(key[u].hash() % (uint32_t)H);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) o[u] = *(volatile int*)&h_owner[h[u]] - 1;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)  // the common case: the first entry holds the key
        found[u] = o[u] >= 0 && GroupKey<kWhat>(a, it.b + o[u]) == key[u] ? h[u] : -1;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = k0 + u * kGroupThreads;
        if (k < it.k1 && found[u] < 0) {
          int hh = h[u];
          for (int probe = 0; probe < H; ++probe, hh = hh + 1 == H ? 0 : hh + 1) {
            int ow = *(volatile int*)&h_owner[hh] - 1;
            if (ow < 0) {
              ow = atomicCAS(&h_owner[hh], 0, k + 1) - 1;
              if (ow < 0) {
                found[u] = hh;  // claimed: a new group
                list[atomicAdd(&a.list_n[it.slot], 1)] = hh;
                break;
              }
            }
            if (GroupKey<kWhat>(a, it.b + ow) == key[u]) {
              found[u] = hh;
              break;
            }
          }
          // H = 2m entries for at most m keys: a probe always ends
        }
        if (k < it.k1) {
          const unsigned act = __activemask(), same = __match_any_sync(act, found[u]);
          if ((threadIdx.x & 31) == __ffs(same) - 1) {
            atomicAdd(&h_cnt[found[u]], __popc(same));
            atomicMax(&h_first[found[u]], 0x7fffffff - k);  // the lowest lane holds the lowest k
          }
          a.id[it.b + k] = found[u];
        }
      }
    }
    if (!last_item(a, it, &s_last)) continue;
    // ---- the slot's last item is in: number the groups ----
    // read through L2: other blocks wrote these
    int ng = __ldcg(&a.list_n[it.slot]);
    int* s_list = s_buf;
    int* s_first = s_buf + kGroupList;
    if (ng <= kGroupList) {
      for (int e = threadIdx.x; e < ng; e += kGroupThreads) {
        const int hh = __ldcg(&list[e]);
        s_list[e] = hh;
        s_first[e] = 0x7fffffff - __ldcg(&h_first[hh]);
      }
      __syncthreads();
      for (int e = threadIdx.x; e < ng; e += kGroupThreads) {
        const int f = s_first[e], hh = s_list[e];
        int r = 0;
        for (int u = 0; u < ng; ++u) r += s_first[u] < f;
        h_rank[hh] = r;
        a.rep[it.t0 + r] = it.b + f;
        a.cnt[it.t0 + r] = __ldcg(&h_cnt[hh]);
        a.pos[it.t0 + r] = a.X[it.b + f];
        if constexpr (kWhat == kGroupsXsph) {
          a.aux[it.t0 + r] = a.V[it.b + f];
          a.sum[it.t0 + r].w = a.rho[it.b + f];
        }
      }
    } else {
      ng = 0;
      for (int k0 = 0; k0 < it.m; k0 += kGroupThreads) {
        const int k = k0 + threadIdx.x;
        const int hh = k < it.m ? __ldcg(&a.id[it.b + k]) : 0;
        const bool first = k < it.m && 0x7fffffff - __ldcg(&h_first[hh]) == k;
        int total;
        const int r = ng + block_scan(first, sh, total);
        if (first) {
          h_rank[hh] = r;
          a.rep[it.t0 + r] = it.b + k;
          a.cnt[it.t0 + r] = __ldcg(&h_cnt[hh]);
          a.pos[it.t0 + r] = a.X[it.b + k];
          if constexpr (kWhat == kGroupsXsph) {
            a.aux[it.t0 + r] = a.V[it.b + k];
            a.sum[it.t0 + r].w = a.rho[it.b + k];
          }
        }
        ng += total;
      }
    }
    __syncthreads();
    // clear the claimed entries for the next pass (h_rank stays: the sums read it)
    const int claimed = __ldcg(&a.list_n[it.slot]);
    for (int e = threadIdx.x; e < claimed; e += kGroupThreads) {
      const int hh = __ldcg(&list[e]);
      h_owner[hh] = 0;
      h_cnt[hh] = 0;
      h_first[hh] = 0;
    }
    if (threadIdx.x == 0) {
      a.ng[it.slot] = ng;
      a.list_n[it.slot] = 0;
      a.done[it.slot] = 0;
    }
    __syncthreads();
  }
}

// Deviation of particle j (cell-relative k) from its group's first particle,
// component c: lambda (kGroupsLambda) or velocity (kGroupsXsph).
template <int kWhat>
__device__ __forceinline__ float group_dev(const GroupArgs& a, const Item& it, int k, int g, int c) {
  if constexpr (kWhat == kGroupsLambda) {
    return dev_from(a.lambda[it.b + k], a.lambda[a.rep[it.t0 + g]]);
  } else {
    const float4 v = a.V[it.b + k], r = a.aux[it.t0 + g];
    return c == 0 ? dev_from(v.x, r.x) : (c == 1 ? dev_from(v.y, r.y) : dev_from(v.z, r.z));
  }
}

// Fixed-point sums over each group of (value - the group's first particle's
// value), two kernels.  group_devmax: the largest |deviation| per group
// (atomicMax on the float bits; +inf marks a non-finite deviation); the last
// block of a slot sets ng = -1 on a non-finite one and zero[slot] when every
// deviation is 0.  k_group_devsum: each deviation scaled by 2^sh, sh from the
// group's bound max|dev| * count < 2^62, added as a 64-bit integer (order-
// free, exact to 2^-62 of the bound); the last block writes the sums
// (lambda: sum = (lambda_rep, sum dev); xsph: sum.xyz) and clears gmax / acc.
template <int kWhat>
__device__ __forceinline__ void group_devmax(const GroupArgs& a) {
  constexpr int C = kWhat == kGroupsLambda ? 1 : 3;
  __shared__ int s_last, s_flag;
  const int items = (int)a.flags[kGroupItems];
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const Item it = item_of(a, item);
    const int* h_rank = a.hash + 2 * it.t0 + 6 * a.np;
    const bool grouped = a.ng[it.slot] > 0;
    for (int k = it.k0 + threadIdx.x; grouped && k < it.k1; k += kGroupThreads) {
      const int g = h_rank[a.id[it.b + k]];
      float d = 0.f;
      bool fin = true;
      for (int c = 0; c < C; ++c) {
        const float e = group_dev<kWhat>(a, it, k, g, c);
        fin &= isfinite(e);
        d = fmaxf(d, fabsf(e));
      }
      const unsigned bits = fin ? __float_as_uint(d) : 0x7f800000u;
      const unsigned act = __activemask(), same = __match_any_sync(act, g);
      const unsigned mx = __reduce_max_sync(same, bits);
      if ((threadIdx.x & 31) == __ffs(same) - 1 && mx) atomicMax(&a.gmax[it.t0 + g], mx);
    }
    if (!last_item(a, it, &s_last)) continue;
    const int ng = a.ng[it.slot];
    if (threadIdx.x == 0) s_flag = 0;
    __syncthreads();
    for (int g = threadIdx.x; g < ng; g += kGroupThreads) {
      const unsigned mx = __ldcg(&a.gmax[it.t0 + g]);
      if (!isfinite(__uint_as_float(mx))) atomicOr(&s_flag, 1);
      if (mx) atomicOr(&s_flag, 2);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (s_flag & 1) a.ng[it.slot] = -1;
      a.zero[it.slot] = !(s_flag & 2);
      a.done[it.slot] = 0;
    }
    if (s_flag & 1)  // ungrouped: clear the bounds now (devsum skips the slot)
      for (int g = threadIdx.x; g < ng; g += kGroupThreads) a.gmax[it.t0 + g] = 0u;
    __syncthreads();
  }
}

template <int kWhat>
__device__ __forceinline__ void group_devsum(const GroupArgs& a) {
  constexpr int C = kWhat == kGroupsLambda ? 1 : 3;
  __shared__ int s_last;
  const int items = (int)a.flags[kGroupItems];
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const Item it = item_of(a, item);
    const int* h_rank = a.hash + 2 * it.t0 + 6 * a.np;
    const bool add = a.ng[it.slot] > 0 && !a.zero[it.slot];
    for (int k = it.k0 + threadIdx.x; add && k < it.k1; k += kGroupThreads) {
      const int g = h_rank[a.id[it.b + k]];
      const float mx = __uint_as_float(a.gmax[it.t0 + g]);
      int e = 0;
      if (mx > 0.f) frexpf(mx, &e);                            // mx < 2^e
      const int sh = 62 - e - (32 - __clz(a.cnt[it.t0 + g]));  // |sum| 2^sh < 2^62
      const unsigned act = __activemask(), same = __match_any_sync(act, g);
      for (int c = 0; c < C; ++c) {
        // |dev| 2^sh < 2^62 is a float without overflow; the scaling is exact
        long long q = __float2ll_rn(ldexpf(group_dev<kWhat>(a, it, k, g, c), sh));
        if (same == 0xffffffffu) {  // a full warp of one group; integer sums: any order, same result
          for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
          if ((threadIdx.x & 31) == 0 && q) atomicAdd(&a.acc[3 * (it.t0 + g) + c], (unsigned long long)q);
        } else if (q) {
          atomicAdd(&a.acc[3 * (it.t0 + g) + c], (unsigned long long)q);
        }
      }
    }
    if (!last_item(a, it, &s_last)) continue;
    const int ng = a.ng[it.slot];
    for (int g = threadIdx.x; g < ng; g += kGroupThreads) {
      const float mx = __uint_as_float(a.gmax[it.t0 + g]);  // from the previous kernel
      int e = 0;
      if (mx > 0.f) frexpf(mx, &e);
      const int sh = 62 - e - (32 - __clz(a.cnt[it.t0 + g]));
      float s3[3];
      for (int c = 0; c < C; ++c) {
        s3[c] = (float)ldexp((double)(long long)__ldcg(&a.acc[3 * (it.t0 + g) + c]), -sh);
        a.acc[3 * (it.t0 + g) + c] = 0ull;
      }
      a.gmax[it.t0 + g] = 0u;
      if constexpr (kWhat == kGroupsLambda) {
        a.sum[it.t0 + g] = make_float4(a.lambda[a.rep[it.t0 + g]], s3[0], 0.f, 0.f);
      } else {
        float4& s4 = a.sum[it.t0 + g];
        s4.x = s3[0], s4.y = s3[1], s4.z = s3[2];
      }
    }
    if (threadIdx.x == 0) a.done[it.slot] = 0;
    __syncthreads();
  }
}

template <int kWhat>
__global__ void __launch_bounds__(kGroupThreads) k_group_insert(GroupArgs a) {
  group_insert<kWhat>(a);
}
template <int kWhat>
__global__ void __launch_bounds__(kGroupThreads) k_group_devmax(GroupArgs a) {
  group_devmax<kWhat>(a);
}
template <int kWhat>
__global__ void __launch_bounds__(kGroupThreads) k_group_devsum(GroupArgs a) {
  group_devsum<kWhat>(a);
}

// ---- work lists: one computing particle per position group -----------------------------

static_assert(kWorkThreads == kGroupThreads, "the work-list kernels use the group kernels' block scan");

// Marks the followers of the current position groups (the group tables the
// lambda pass of this iteration just built): follow[i] = the group's first
// particle when particle i of a grouped cell is not that particle, else -1;
// blocks[b] = the computing particles of block b.  The block that finishes
// last turns blocks[] into exclusive offsets (so the list is in cell order).
struct WorkArgs {
  const uint32_t* skeys;
  const uint32_t* cell_flags;
  const int* grp_n;
  const int* grp_off;
  const int* grp_id;
  const int* grp_hash;
  const int* grp_rep;
  int np, n;
  int* follow;
  int* blocks;
  int* list;
  uint32_t* flags;
};

// Returns whether the thread's particle computes (with groups).
__device__ __forceinline__ bool work_mark(const WorkArgs& w) {
  uint32_t* flags = w.flags;
  int* blocks = w.blocks;
  const int n = w.n, np = w.np;
  __shared__ int sh[80];
  __shared__ int s_last;
  if (flags[kGroupCount] == 0u) {  // no grouped cell this step: every particle computes, in order
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      flags[kWorkCount] = (uint32_t)n;
      flags[kWorkIdentity] = 1u;
    }
    return false;
  }
  const int i = blockIdx.x * kWorkThreads + threadIdx.x;
  int r = -1;
  if (i < n) {
    const uint32_t sl = w.cell_flags[w.skeys[i]] >> kCellSlotShift;
    if (sl) {
      const int slot = (int)sl - 1;
      if (w.grp_n[slot] > 0) {
        // the particle's hash entry -> its group's rank -> the group's first particle
        const int t0 = w.grp_off[slot];
        const int rank = w.grp_hash[2 * t0 + 6 * np + w.grp_id[i]];
        const int rep = w.grp_rep[t0 + rank];
        if (rep != i) r = rep;
      }
    }
    w.follow[i] = r;
  }
  const int cnt = __syncthreads_count(i < n && r < 0);
  if (threadIdx.x == 0) blocks[blockIdx.x] = cnt;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&flags[kWorkDone], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return i < n && r < 0;
  __threadfence();
  // the last block: exclusive offsets of every block, in chunks of kWorkThreads
  int carry = 0;
  for (int b0 = 0; b0 < (int)gridDim.x; b0 += kWorkThreads) {
    const int b = b0 + threadIdx.x;
    const int v = b < (int)gridDim.x ? __ldcg(&blocks[b]) : 0;
    int total;
    const int ex = block_scan_value(v, sh, total);
    if (b < (int)gridDim.x) blocks[b] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    flags[kWorkCount] = (uint32_t)carry;
    flags[kWorkDone] = 0u;
  }
  return i < n && r < 0;
}

// list[blocks[b] + rank] = i for the computing particles of block b, in order.
__device__ __forceinline__ void work_list(const WorkArgs& w) {
  __shared__ int sh[80];
  if (w.flags[kWorkIdentity]) return;
  const int i = blockIdx.x * kWorkThreads + threadIdx.x;
  const bool keep = i < w.n && w.follow[i] < 0;
  int total;
  const int rank = block_scan(keep, sh, total);
  if (keep) w.list[w.blocks[blockIdx.x] + rank] = i;
}

__global__ void __launch_bounds__(kWorkThreads) k_work_mark(WorkArgs w) { work_mark(w); }
__global__ void __launch_bounds__(kWorkThreads) k_work_list(WorkArgs w) { work_list(w); }

// The followers take their group's results.
template <int kKind>
__device__ __forceinline__ void follow_group(const PassArgs& a, const int* follow, int i) {
  if (i >= a.n || a.flags[kWorkIdentity]) return;
  const int r = follow[i];
  if (r < 0) return;
  if constexpr (kKind == kLambda) {
    a.lambda[i] = a.lambda[r];
    a.rho[i] = a.rho[r];
    a.XL[i] = a.XL[r];  // the same position
  } else if constexpr (kKind == kDeltaP) {
    const float4 t = a.T[r];
    a.T[i] = t;
    put_components(a.S_out, a.stride, i, t);
  } else {
    // DeltaPPass<true>::finish with the group's final position
    const float4 xf = a.npos[r];
    const float4 x0 = a.xs[i];
    a.npos[i] = make_float4(xf.x, xf.y, xf.z, x0.w);
    put_components(a.S_out, a.stride, i, xf);
    const float4 v = make_float4((xf.x - x0.x) * a.c.inv_dt, (xf.y - x0.y) * a.c.inv_dt,
                                 (xf.z - x0.z) * a.c.inv_dt, 0.f);
    a.vel[i] = v;
    a.VR[i] = make_float4(v.x, v.y, v.z, a.rho[i]);
    if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z)) {
      atomicOr(&a.cell_flags[a.skeys[i]], (uint32_t)kCellVelNonFinite);
      atomicOr(&a.flags[kFlagXsphExact], 1u);
    }
    a.pos[i] = x0;
    a.iid[i] = a.iid_s[i];
  }
}

template <int kKind>
__global__ void __launch_bounds__(256) k_follow(PassArgs a, const int* __restrict__ follow) {
  follow_group<kKind>(a, follow, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---- current-cell order ---------------------------------------------------------------

// The pass's computing particles (its list, or every particle) by the cell
// they are in now: count (integer atomics: the counts are exact, the rank
// inside a cell is arbitrary), exclusive scan over cells, scatter.  Consecutive
// particles of the resulting list mostly share a window, so a warp's lanes
// load the same candidates and run similar loops.  A particle's result does
// not depend on its place in the list (sparse / dense routing is per
// particle), so the arbitrary ranks leave results bitwise reproducible.
// t: a slot of the pass's list (its particle i), or any beyond it (i unused).
__device__ __forceinline__ void bucket_count(const PassArgs& a, int t, int i, uint32_t* bcnt, uint2* bent) {
  const SceneGeom g = geom_of(a.c, a.G, i);
  const int3 q = cell_of(a.c, g, a.X[i]);
  const uint32_t cell = (uint32_t)cell_index(g, q.x, q.y, q.z);
  // one atomic per cell and warp (particles piled into a cell share it)
  const unsigned act = __activemask();
  const unsigned same = __match_any_sync(act, cell);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  uint32_t base = 0u;
  if (lane == leader) base = atomicAdd(&bcnt[cell], (uint32_t)__popc(same));
  base = __shfl_sync(same, base, leader);
  bent[t] = make_uint2(cell, base + (uint32_t)__popc(same & ((1u << lane) - 1u)));
}

__global__ void __launch_bounds__(256) k_bucket_count(PassArgs a, uint32_t* __restrict__ bcnt,
                                                      uint2* __restrict__ bent) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < work_count(a)) bucket_count(a, t, work_particle(a, t), bcnt, bent);
}

// bstart: the prefix of the counts, or where a.paired of pair_slots of them (the
// slots left over hold -1).
__global__ void __launch_bounds__(256) k_bucket_scatter(PassArgs a, const uint32_t* __restrict__ bcnt,
                                                        const uint32_t* __restrict__ bstart,
                                                        const uint2* __restrict__ bent, int* __restrict__ bucket) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) a.flags[kBucketCount] = bstart[a.c.cells];
  if (t >= work_count(a)) return;
  const uint2 e = bent[t];
  const bool apart = a.paired && a.flags[kGroupCount] != 0u;
  const uint32_t slot = bstart[e.x] + (apart ? 2u * e.y : e.y);
  bucket[slot] = work_particle(a, t);
  if (a.paired && (apart || ((e.y & 1u) == 0u && e.y + 1u == bcnt[e.x]))) bucket[slot + 1u] = -1;
}

GroupArgs group_args(const StepConsts& c, const SolverScratch& s, const float4* X, const float4* V, int n) {
  GroupArgs a;
  a.chunk = group_chunk(c, n);
  a.X = X;
  a.V = V;
  a.rho = s.rho;
  a.lambda = s.lambda;
  a.cs = s.cell_start;
  a.flags = s.flags;
  a.n = n;
  a.np = s.grp_pool;
  a.cell = s.grp_cell;
  a.off = s.grp_off;
  a.item_off = s.grp_item_off;
  a.item_slot = s.grp_item_slot;
  a.done = s.grp_done;
  a.ng = s.grp_n;
  a.rep = s.grp_rep;
  a.cnt = s.grp_cnt;
  a.pos = s.grp_pos;
  a.sum = s.grp_sum;
  a.aux = s.grp_aux;
  a.id = s.grp_id;
  a.hash = s.grp_hash;
  a.list = s.grp_list;
  a.list_n = s.grp_list_n;
  a.gmax = s.grp_max;
  a.acc = s.grp_acc;
  a.zero = s.grp_zero;
  return a;
}

// Whether the lambda / delta_p passes run on work lists (groups exist only
// from kGroupCell particles on, and the zero gradient of co-located particles
// needs kernel_eps > 0).
bool use_work_list(const StepConsts& c, int n) { return n >= kGroupCell && c.keps2 > 0.f; }

WorkArgs work_args(const SolverScratch& s, int n) {
  return WorkArgs{s.keys_sorted, s.cell_flags, s.grp_n, s.grp_off, s.grp_id,      s.grp_hash,    s.grp_rep,
                  s.grp_pool,    n,            s.work_follow, s.work_blocks, s.work_list, s.flags};
}

// ---- small steps: the work around a pass in one launch -----------------------------------
//
// A step of a few thousand particles spends its time in launches (2 us each,
// whatever they do): group tables, work list, followers and buckets took 13 of
// the 15 launches of an iteration.  In a small step (is_small: every particle
// dense, one 1,024-thread block per 1,024 particles fits on the chip at once)
// everything between two passes is one cooperative launch, its phases separated
// by grid barriers and skipped where the step has no grouped cells:
//   k_small_before   (lambda, xsph)  the followers of the last delta_p pass, the
//                    position (xsph: position and density) groups, the work list,
//                    the buckets
//   k_small_between  (delta_p)       the lambda pass's followers, the sums of
//                    lambda
// The buckets are built only where they matter: when more than one computing
// particle in kMovedShare has left its grid cell (the delta_p passes count
// them); else the passes take the particles (with groups, the work list) in grid
// order, which is then nearly the current cells' (the order changes no result).
// A step: 253 -> 99 us (1,728 particles), 268 -> 113 (8,000), 717 -> 706 (126,976,
// three quarters of them on six points; 737 with a barrier after each of the
// phases and every list bucketed).

constexpr int kMovedShare = 8;

// Every block of the (cooperative) grid arrives before any goes on; writes
// before it are visible after it.  Bounded: a block that has polled `polls`
// times, or finds that another one gave up, records kErrBarrierTimeout and
// returns false (its caller returns).  A block goes past a barrier only when
// every block has reached it, so what it reads there is complete; the block that
// gave up is missing at the next one, where the others give up too.  The step's
// later kernels then do nothing (kStepFailed): they read lists that were not
// finished, and would count this kernel's arrivals as theirs.
__device__ __forceinline__ bool grid_barrier(uint32_t* flags, int polls) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile uint32_t* gen = &flags[kBarrierGen];
    const uint32_t g = *gen;
    int ok = 1;
    __threadfence();
    if (atomicAdd(&flags[kBarrierCount], 1u) == gridDim.x - 1) {
      flags[kBarrierCount] = 0u;
      __threadfence();
      atomicAdd(&flags[kBarrierGen], 1u);
    } else {
      volatile uint32_t* failed = &flags[kStepFailed];
      for (int k = 1; ok && *gen == g; ++k) ok = k < polls && ((k & 63) != 0 || *failed == 0u);
      if (!ok) {
        atomicOr(&flags[kErrorWord], (uint32_t)kErrBarrierTimeout);
        *failed = 1u;
        flags[kDirtyWord] = 1u;
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

struct SmallArgs {
  PassArgs p;        // the pass that follows
  GroupArgs g;
  WorkArgs w;
  uint32_t* bcnt;
  uint32_t* bstart;
  uint2* bent;
  int* bucket;
  uint32_t* bpart;
  int iteration;     // of the pass (xsph: niter)
  int groups;        // the step may have grouped cells
  int buckets;       // current-cell order is on
};

// Whether an earlier kernel of the step gave up (one answer for the block).
__device__ __forceinline__ bool step_failed(const uint32_t* flags) {
  return __syncthreads_or(*(volatile const uint32_t*)&flags[kStepFailed] != 0u) != 0;
}

// kLast: the delta_p pass whose followers come first (kDeltaPFinal: xsph follows).
template <int kLast>
__global__ void __launch_bounds__(kWorkThreads, 1) k_small_before(SmallArgs a) {
  constexpr bool kXsphNext = kLast == kDeltaPFinal;
  uint32_t* flags = a.p.flags;
  const int i = blockIdx.x * kWorkThreads + threadIdx.x;
  const int n = a.p.n;
  const bool groups = a.groups && flags[kGroupCount] != 0u;
  const uint32_t moved = a.buckets && a.iteration > 0 ? flags[kMoved0 + ((a.iteration + 1) & 1)] : 0u;
  const bool buckets = a.buckets && moved > (uint32_t)n / kMovedShare;  // uniform over the grid
  const int polls = a.p.c.wait_polls;
  if ((groups || buckets) && step_failed(flags)) return;
  const int cells1 = a.p.c.cells + 1;
  if (buckets)
    for (int k = i; k < cells1; k += gridDim.x * kWorkThreads) a.bcnt[k] = 0u;
  bool computes = i < n;
  if (groups) {
    if (a.iteration > 0) {
      follow_group<kLast>(a.p, a.w.follow, i);
      if (!grid_barrier(flags, polls)) return;
    }
    if constexpr (kXsphNext) {
      group_insert<kGroupsXsph>(a.g);
      if (!grid_barrier(flags, polls)) return;
      group_devmax<kGroupsXsph>(a.g);
      if (!grid_barrier(flags, polls)) return;
      group_devsum<kGroupsXsph>(a.g);
    } else {
      group_insert<kGroupsPos>(a.g);
      if (!grid_barrier(flags, polls)) return;
      computes = work_mark(a.w);
      if (!buckets) {
        if (!grid_barrier(flags, polls)) return;
        work_list(a.w);
      }
    }
  } else {
    if (!kXsphNext && i == 0) {
      flags[kWorkCount] = (uint32_t)n;
      flags[kWorkIdentity] = 1u;
    }
    if (buckets && !grid_barrier(flags, polls)) return;
  }
  if (!a.buckets) return;
  const bool listed = groups && !kXsphNext;
  // the count this iteration's delta_p pass adds to (the last one's was read above)
  if (i == 0) {
    flags[kMoved0 + (a.iteration & 1)] = 0u;
    flags[kBucketIdentity] = !buckets && !listed;
    if (!listed) flags[kBucketCount] = (uint32_t)n;
    else if (!buckets) flags[kBucketCount] = flags[kWorkCount];  // (complete since the barrier)
  }
  if (!buckets) return;
  // count, exclusive scan over the cells (every block a share), scatter
  if (computes) bucket_count(a.p, i, i, a.bcnt, a.bent);
  if (!grid_barrier(flags, polls)) return;
  __shared__ int sh[80];
  const int per_block = (cells1 + (int)gridDim.x - 1) / (int)gridDim.x;
  const int per_thread = (per_block + kWorkThreads - 1) / kWorkThreads;
  const int end = min((int)(blockIdx.x + 1) * per_block, cells1);
  const int from = min((int)blockIdx.x * per_block + (int)threadIdx.x * per_thread, end);
  const int to = min(from + per_thread, end);
  int sum = 0;
  for (int k = from; k < to; ++k) sum += (int)a.bcnt[k];
  int total;
  int run = block_scan_value(sum, sh, total);
  if (threadIdx.x == 0) a.bpart[blockIdx.x] = (uint32_t)total;
  if (!grid_barrier(flags, polls)) return;
  int before;  // the sum of the blocks before this one
  block_scan_value(threadIdx.x < blockIdx.x ? (int)a.bpart[threadIdx.x] : 0, sh, before);
  run += before;
  for (int k = from; k < to; ++k) {
    a.bstart[k] = (uint32_t)run;
    run += (int)a.bcnt[k];
  }
  if (!grid_barrier(flags, polls)) return;
  if (listed && i == 0) flags[kBucketCount] = flags[kWorkCount];
  if (computes) {
    const uint2 e = a.bent[i];
    a.bucket[a.bstart[e.x] + e.y] = i;
  }
}

__global__ void __launch_bounds__(kWorkThreads, 1) k_small_between(SmallArgs a) {
  const int polls = a.p.c.wait_polls;
  if (a.p.flags[kGroupCount] == 0u || step_failed(a.p.flags)) return;
  follow_group<kLambda>(a.p, a.w.follow, blockIdx.x * kWorkThreads + threadIdx.x);
  if (!grid_barrier(a.p.flags, polls)) return;
  group_devmax<kGroupsLambda>(a.g);
  if (!grid_barrier(a.p.flags, polls)) return;
  group_devsum<kGroupsLambda>(a.g);
}

// Points a small step's pass at its particles: the buckets, or the work list.
void small_list(PassArgs& a, const SolverScratch& s, bool xsph) {
  a.paired = 0;
  if (a.c.order) {
    a.list = s.bucket;
    a.count_word = kBucketCount;
    a.identity_word = kBucketIdentity;
  } else if (!xsph && use_work_list(a.c, a.n)) {
    a.list = s.work_list;  // with its own count and identity
  }
}

SmallArgs small_args(const PassArgs& p, const SolverScratch& s, const float4* X, int pass) {
  SmallArgs a;
  a.p = p;
  a.g = group_args(p.c, s, X, p.V, p.n);
  a.w = work_args(s, p.n);
  if (p.c.order) a.w.list = s.bucket;  // where the passes look
  a.bcnt = s.bcnt, a.bstart = s.bstart, a.bent = s.bent, a.bucket = s.bucket, a.bpart = s.bpart;
  a.iteration = pass / 2;
  a.groups = p.n >= kGroupCell && p.c.keps2 > 0.f;
  a.buckets = p.c.order;
  return a;
}

template <class Kernel>
cudaError_t launch_cooperative(Kernel kernel, const SmallArgs& a, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.p.n + kWorkThreads - 1) / kWorkThreads);
  cfg.blockDim = dim3(kWorkThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Before a lambda pass (kLast = kDeltaP) or the xsph pass (kDeltaPFinal): see
// k_small_before.  The first lambda pass has no followers and its particles are
// in their grid cells, so without groups there is nothing to launch but the
// identity's flags, which a step clears to "no identity".
template <int kLast>
cudaError_t small_before(PassArgs& a, const SolverScratch& s, int pass, cudaStream_t stream) {
  constexpr bool kXsphNext = kLast == kDeltaPFinal;
  SmallArgs args = small_args(a, s, a.X, pass);
  if constexpr (!kXsphNext) {
    // the delta_p pass before wrote X (its T) and its component copy
    args.p.T = const_cast<float4*>(a.X);
    args.p.S_out = const_cast<float*>(a.S);
  }
  const bool first = args.iteration == 0;
  if (!args.groups && (first || !args.buckets)) return cudaSuccess;  // every particle, in order (a.list is null)
  small_list(a, s, kXsphNext);
  return launch_cooperative(k_small_before<kLast>, args, stream);
}

cudaError_t small_between(PassArgs& a, const SolverScratch& s, int pass, cudaStream_t stream) {
  const SmallArgs args = small_args(a, s, nullptr, pass);
  const bool first = args.iteration == 0;
  if (args.groups || !(first || !args.buckets)) small_list(a, s, false);  // as its lambda pass
  if (args.buckets) a.moved_word = kMoved0 + (args.iteration & 1);
  return args.groups ? launch_cooperative(k_small_between, args, stream) : cudaSuccess;
}

// kGroupsPos: the lambda pass's groups.  kGroupsLambda: their lambda sums for
// delta_p.  kGroupsXsph: the (position, density) groups and velocity sums.
template <int kWhat>
cudaError_t launch_groups(const StepConsts& c, const SolverScratch& s, const float4* X, const float4* V, int n,
                          cudaStream_t stream) {
  if (n < kGroupCell) return cudaSuccess;  // no cell can hold kGroupCell particles
  const GroupArgs a = group_args(c, s, X, V, n);
  const int grid = c.dense_grid;
  if constexpr (kWhat != kGroupsLambda) k_group_insert<kWhat><<<grid, kGroupThreads, 0, stream>>>(a);
  if constexpr (kWhat != kGroupsPos) {
    k_group_devmax<kWhat><<<grid, kGroupThreads, 0, stream>>>(a);
    k_group_devsum<kWhat><<<grid, kGroupThreads, 0, stream>>>(a);
  }
  return cudaGetLastError();
}

PassArgs base_args(const StepConsts& c, const Geometry& G, const float4* X, const uint32_t* cs,
                   int n, const SolverScratch& s, int pass) {
  PassArgs a = {};
  a.c = c;
  a.G = G;
  a.X = X;
  a.cs = cs;
  a.n = n;
  a.dense_all = dense_for_all(c, n);
  a.counter = kDenseCount0 + (pass & 1);
  a.next_counter = kDenseCount0 + ((pass + 1) & 1);
  a.item_counter = kItemCount0 + (pass & 1);
  a.next_item_counter = kItemCount0 + ((pass + 1) & 1);
  a.flags = s.flags;
  a.dense = s.dense;
  // a position buffer's component copy: sa beside xa, sb beside xb; the final
  // positions' beside the buffer that is free then
  a.stride = s.stride;
  a.hits = s.hits;
  a.hit_n = s.hit_n;
  a.hit_stride = s.hit_stride;
  a.XL = s.xl;
  a.cell_flags = s.cell_flags;
  a.skeys = s.keys_sorted;
  a.lambda = s.lambda;
  a.rho = s.rho;
  a.grp_off = s.grp_off;
  a.grp_n = s.grp_n;
  a.grp_cnt = s.grp_cnt;
  a.grp_pos = s.grp_pos;
  a.grp_sum = s.grp_sum;
  a.grp_aux = s.grp_aux;
  a.count_word = kWorkCount;
  a.identity_word = kWorkIdentity;
  a.moved_word = -1;
  return a;
}

// Whether the sparse kernel takes two particles a thread where the passes take
// the buckets: not with a kernel_eps that leaves it no packed walk (fast_hits),
// where the two would be walked one after the other (kernel_eps 0, 262,144
// particles: a step 922 us in pairs, 894 the other way).
bool takes_pairs(const StepConsts& c) { return c.keps2 >= kNormalMin; }

// The pass takes the buckets (the delta_p passes of an iteration those of its
// lambda pass: the same positions).
void use_buckets(PassArgs& a, const SolverScratch& s) {
  a.list = s.bucket;
  a.count_word = kBucketCount;
  a.identity_word = -1;
  a.paired = !a.dense_all && takes_pairs(a.c);
}

// Makes the pass take its computing particles in current-cell order: buckets
// them (bucket_launches) and points the pass at the buckets.
cudaError_t bucket_by_cell(PassArgs& a, const SolverScratch& s, int n, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(s.bcnt, 0, sizeof(uint32_t) * (a.c.cells + 1), stream);
  if (e != cudaSuccess) return e;
  const int blocks = (n + 255) / 256;
  a.paired = !a.dense_all && takes_pairs(a.c);
  k_bucket_count<<<blocks, 256, 0, stream>>>(a, s.bcnt, s.bent);
  if ((e = exclusive_scan(s.bcnt, s.bstart, a.c.cells + 1, s.bpart, stream,
                          a.paired ? s.flags + kGroupCount : nullptr)) != cudaSuccess)
    return e;
  k_bucket_scatter<<<blocks, 256, 0, stream>>>(a, s.bcnt, s.bstart, s.bent, s.bucket);
  use_buckets(a, s);
  return cudaGetLastError();
}

template <int kKind>
cudaError_t run_pass(const PassArgs& a, cudaStream_t stream) {
  // the dense kernel's dynamic shared memory: the hit queue (8 bytes per chunk
  // and thread), then the stage
  const size_t dense_queue = (size_t)8 * a.c.queue_dense * kDenseThreads;
  const size_t dense_smem = sizeof(float4) * (size_t)max(a.c.stage_dense, 0);
  const long long slots = a.paired ? 2ll * a.n : a.n;  // of the pass's list, at most
  constexpr bool kPairs = kKind == kLambda || kKind == kXsph;
  const int per_sparse = kPairs && a.paired ? 2 * kSparseThreads : kSparseThreads;
  const int sparse_blocks = (int)((slots + per_sparse - 1) / per_sparse);
  if (a.dense_all) {
    // the sparse kernel has nothing to do
  } else if (kPairs && a.paired) {
    if constexpr (kPairs) k_sparse_pair<kKind><<<sparse_blocks, kSparseThreads, 0, stream>>>(a);
    if constexpr (kKind == kXsph) {
      k_xsph_mark<<<(a.n + 255) / 256, 256, 0, stream>>>(a);
      k_xsph_poison<<<(int)((slots / 2 + 255) / 256), 256, 0, stream>>>(a);
    }
  } else {
    k_sparse<kKind><<<sparse_blocks, kSparseThreads, 0, stream>>>(a);
  }
  // no more blocks than batches where their number is known
  const int per_block = dense_smem ? 1 : kDenseWarps / a.c.dense_split;
  const int grid = a.dense_all ? min(a.c.dense_grid, ((a.n + 31) / 32 + per_block - 1) / per_block) : a.c.dense_grid;
  if (dense_smem)
    k_dense<kKind, true><<<grid, kDenseThreads, dense_queue + dense_smem, stream>>>(a);
  else
    k_dense<kKind, false><<<grid, kDenseThreads, dense_queue, stream>>>(a);
  return cudaGetLastError();
}

template <int kKind>
cudaError_t allow_stage(int queue, int stage) {
  cudaError_t e = cudaFuncSetAttribute(k_dense<kKind, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, queue);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_dense<kKind, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, queue + stage);
  return e;
}

}  // namespace

// Lets the dense kernels take their largest hit queue, and the staged ones up to
// kStageMax staged slots of dynamic shared memory (the current device; call
// before any capture).
cudaError_t set_pass_kernel_attributes() {
  const int queue = 8 * kMaxQueueDense * kDenseThreads;
  const int stage = (int)sizeof(float4) * kStageMax;
  cudaError_t e = allow_stage<kLambda>(queue, stage);
  if (e == cudaSuccess) e = allow_stage<kDeltaP>(queue, stage);
  if (e == cudaSuccess) e = allow_stage<kDeltaPFinal>(queue, stage);
  if (e == cudaSuccess) e = allow_stage<kXsph>(queue, stage);
  return e;
}

ClearList step_clears(const StepConsts& c, const SolverScratch& s) {
  // (the group tables as alloc_groups leaves them)
  const size_t np = (size_t)s.grp_pool, slots = group_slots(s.grp_pool);
  return ClearList{{s.cell_flags, s.flags, nullptr},
                   {c.cells + 1, kNumFlags, 0},
                   s.flags + kDirtyWord,
                   {(uint32_t*)s.grp_hash, (uint32_t*)s.grp_max, (uint32_t*)s.grp_acc, (uint32_t*)s.grp_list_n,
                    (uint32_t*)s.grp_done},
                   {8 * np, np, 6 * np, slots, slots}};
}

cudaError_t reorder(const StepConsts& c, const uint32_t* perm, const float4* pos, const float4* vel,
                    const uint32_t* iid, int n, SolverScratch& s, cudaStream_t stream) {
  k_reorder<<<(n + 255) / 256, 256, 0, stream>>>(perm, pos, vel, iid, n, c, s.xs, s.xa,
                                                  s.sa, s.stride, s.iid_s, s.flags, s.keys_sorted, s.cell_start, s.cell_flags,
                                                  s.grp_cell, s.grp_off, s.grp_item_off, s.grp_item_slot,
                                                  group_chunk(c, n));
  return cudaGetLastError();
}

namespace {

cudaError_t launch_work_list(const SolverScratch& s, int n, cudaStream_t stream) {
  const int blocks = (n + kWorkThreads - 1) / kWorkThreads;
  const WorkArgs w = work_args(s, n);
  k_work_mark<<<blocks, kWorkThreads, 0, stream>>>(w);
  k_work_list<<<blocks, kWorkThreads, 0, stream>>>(w);
  return cudaGetLastError();
}

template <int kKind>
cudaError_t launch_follow(const PassArgs& a, const SolverScratch& s, cudaStream_t stream) {
  k_follow<kKind><<<(a.n + 255) / 256, 256, 0, stream>>>(a, s.work_follow);
  return cudaGetLastError();
}

// The component copy of position buffer X.
float* components_of(const SolverScratch& s, const float4* X) { return X == s.xa ? s.sa : s.sb; }

}  // namespace

// A step whose work around the passes runs in cooperative launches
// (k_small_before): every particle dense and one block per kWorkThreads
// particles on an SM of its own.
bool is_small(const StepConsts& c, int n) {
  return dense_for_all(c, n) && n < kDenseAllBelow &&
         (n + kWorkThreads - 1) / kWorkThreads <= c.dense_grid / kDenseBlocksPerSm;
}

cudaError_t launch_lambda(const StepConsts& c, const Geometry& G, const float4* X, const uint32_t* cs, int n,
                          const SolverScratch& s, int pass, cudaStream_t stream) {
  if (is_small(c, n)) {
    PassArgs a = base_args(c, G, X, cs, n, s, pass);
    a.S = components_of(s, X);
    const cudaError_t e = small_before<kDeltaP>(a, s, pass, stream);
    return e == cudaSuccess ? run_pass<kLambda>(a, stream) : e;
  }
  cudaError_t e = launch_groups<kGroupsPos>(c, s, X, nullptr, n, stream);
  if (e != cudaSuccess) return e;
  const bool wl = use_work_list(c, n);
  if (wl && (e = launch_work_list(s, n, stream)) != cudaSuccess) return e;
  PassArgs a = base_args(c, G, X, cs, n, s, pass);
  a.S = components_of(s, X);
  if (wl) a.list = s.work_list;
  if (c.order && (e = bucket_by_cell(a, s, n, stream)) != cudaSuccess) return e;
  if ((e = run_pass<kLambda>(a, stream)) != cudaSuccess) return e;
  return wl ? launch_follow<kLambda>(a, s, stream) : cudaSuccess;
}

cudaError_t launch_delta_p(const StepConsts& c, const Geometry& G, const float4* X, const uint32_t* cs, int n,
                           const SolverScratch& s, int pass, float4* T, cudaStream_t stream) {
  PassArgs a = base_args(c, G, s.xl, cs, n, s, pass);  // X with its lambda
  a.S = components_of(s, X);
  a.S_out = components_of(s, T);
  a.T = T;
  if (is_small(c, n)) {
    const cudaError_t e = small_between(a, s, pass, stream);
    return e == cudaSuccess ? run_pass<kDeltaP>(a, stream) : e;
  }
  cudaError_t e = launch_groups<kGroupsLambda>(c, s, X, nullptr, n, stream);
  if (e != cudaSuccess) return e;
  const bool wl = use_work_list(c, n);
  if (wl) a.list = s.work_list;
  if (c.order) use_buckets(a, s);
  if ((e = run_pass<kDeltaP>(a, stream)) != cudaSuccess) return e;
  return wl ? launch_follow<kDeltaP>(a, s, stream) : cudaSuccess;
}

cudaError_t launch_delta_p_final(const StepConsts& c, const Geometry& G, const float4* X, const uint32_t* cs, int n,
                                 const SolverScratch& s, int pass, float4* pos, float4* npos,
                                 float4* vel, uint32_t* iid, cudaStream_t stream) {
  PassArgs a = base_args(c, G, s.xl, cs, n, s, pass);
  a.S = components_of(s, X);
  a.VR = X == s.xa ? s.xb : s.xa;  // the positions go to npos: T's buffers are free
  a.S_out = components_of(s, a.VR);
  a.xs = s.xs;
  a.iid_s = s.iid_s;
  a.npos = npos;
  a.vel = vel;
  a.pos = pos;
  a.iid = iid;
  if (is_small(c, n)) {
    const cudaError_t e = small_between(a, s, pass, stream);
    return e == cudaSuccess ? run_pass<kDeltaPFinal>(a, stream) : e;
  }
  cudaError_t e = launch_groups<kGroupsLambda>(c, s, X, nullptr, n, stream);
  if (e != cudaSuccess) return e;
  const bool wl = use_work_list(c, n);
  if (wl) a.list = s.work_list;
  if (c.order) use_buckets(a, s);
  if ((e = run_pass<kDeltaPFinal>(a, stream)) != cudaSuccess) return e;
  return wl ? launch_follow<kDeltaPFinal>(a, s, stream) : cudaSuccess;
}

// ---- vorticity confinement ---------------------------------------------------------------

namespace {

// Spiky gradient grad W(r) for kernel_eps <= |r| < h (else zero), r = x_i - x_j.
__device__ __forceinline__ bool spiky_grad(const StepConsts& c, float ex, float ey, float ez, float& gx,
                                           float& gy, float& gz) {
  const float r2 = dist2(ex, ey, ez);
  if (!(r2 < c.h2) || r2 < c.keps2) return false;
  const float ir = rsqrtf(r2);
  const float t = c.h - r2 * ir;
  const float sc = c.spiky_coef * t * t * ir;
  gx = sc * ex, gy = sc * ey, gz = sc * ez;
  return true;
}

struct VortOmega {
  const StepConsts& c;
  const float4* __restrict__ U;
  float4 xi, ui;
  int i;
  float wx = 0.f, wy = 0.f, wz = 0.f;
  __device__ __forceinline__ void visit(float4 xj, int j) {
    float gx, gy, gz;
    if (j == i || !spiky_grad(c, xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, gx, gy, gz)) return;
    const float4 uj = __ldg(U + j);
    const float dx = uj.x - ui.x, dy = uj.y - ui.y, dz = uj.z - ui.z;
    wx += dy * gz - dz * gy;
    wy += dz * gx - dx * gz;
    wz += dx * gy - dy * gx;
  }
};

struct VortEta {
  const StepConsts& c;
  const float4* __restrict__ W;
  float4 xi;
  int i;
  float ex = 0.f, ey = 0.f, ez = 0.f;
  __device__ __forceinline__ void visit(float4 xj, int j) {
    float gx, gy, gz;
    if (j == i || !spiky_grad(c, xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, gx, gy, gz)) return;
    const float m = __ldg(W + j).w;
    ex += m * gx;
    ey += m * gy;
    ez += m * gz;
  }
};

__global__ void __launch_bounds__(128)
k_vort_omega(StepConsts c, Geometry G, const float4* __restrict__ X, const float4* __restrict__ U,
             const uint32_t* __restrict__ cs, int n, float4* __restrict__ W) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = X[i];
  const SceneGeom g = geom_of(c, G, i);
  VortOmega p{c, U, xi, U[i], i};
  visit_window(g, cs, n, cell_of(c, g, xi), FromGlobal{X}, p);
  W[i] = make_float4(p.wx, p.wy, p.wz, sqrtf(dist2(p.wx, p.wy, p.wz)));
}

__global__ void __launch_bounds__(128)
k_vort_force(StepConsts c, Geometry G, const float4* __restrict__ X, const float4* __restrict__ W,
             const uint32_t* __restrict__ cs, int n, float4* __restrict__ U) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 xi = X[i];
  const SceneGeom g = geom_of(c, G, i);
  VortEta p{c, W, xi, i};
  visit_window(g, cs, n, cell_of(c, g, xi), FromGlobal{X}, p);
  const float len = sqrtf(dist2(p.ex, p.ey, p.ez));
  if (!(len > 0.f) || !isfinite(len)) return;
  const float nx = p.ex / len, ny = p.ey / len, nz = p.ez / len;
  const float4 w = W[i];
  const float s = c.dt * c.vort_eps;
  float4 u = U[i];
  u.x += s * (ny * w.z - nz * w.y);
  u.y += s * (nz * w.x - nx * w.z);
  u.z += s * (nx * w.y - ny * w.x);
  U[i] = u;
}

}  // namespace

cudaError_t launch_vorticity(const StepConsts& c, const Geometry& G, const float4* X, const uint32_t* cs, int n,
                             const SolverScratch& s, float4* NV, cudaStream_t stream) {
  const int blocks = (n + 127) / 128;
  k_vort_omega<<<blocks, 128, 0, stream>>>(c, G, X, NV, cs, n, s.xb);
  k_vort_force<<<blocks, 128, 0, stream>>>(c, G, X, s.xb, cs, n, NV);
  return cudaGetLastError();
}

cudaError_t launch_xsph(const StepConsts& c, const Geometry& G, const float4* X, const float4* V, const uint32_t* cs,
                        int n, const SolverScratch& s, int pass, float4* pos, float4* npos, float4* vel,
                        uint32_t* iid, float4* NV, cudaStream_t stream) {
  PassArgs a = base_args(c, G, X, cs, n, s, pass);
  // where the last position update left them: after niter - 1 swaps of xa and
  // xb it read one and used the other
  a.VR = (pass / 2) % 2 ? s.xb : s.xa;
  a.S = components_of(s, a.VR);
  a.V = V;
  a.NV = NV;
  if (is_small(c, n)) {
    // the last position update's followers, as launch_delta_p_final has it
    a.xs = s.xs, a.iid_s = s.iid_s, a.npos = npos, a.vel = vel, a.pos = pos, a.iid = iid;
    a.S_out = components_of(s, a.VR);
    const cudaError_t e = small_before<kDeltaPFinal>(a, s, pass, stream);
    return e == cudaSuccess ? run_pass<kXsph>(a, stream) : e;
  }
  cudaError_t e = launch_groups<kGroupsXsph>(c, s, X, V, n, stream);
  if (e != cudaSuccess) return e;
  if (c.order && (e = bucket_by_cell(a, s, n, stream)) != cudaSuccess) return e;
  return run_pass<kXsph>(a, stream);
}

}  // namespace pbf

namespace pbf {

int pass_launches(const StepConsts& c, int n) {
  return dense_for_all(c, n) ? 1 : 2;
}

// k_xsph_mark and k_xsph_poison.
int poison_launches(const StepConsts& c, int n) {
  return c.order && !dense_for_all(c, n) && takes_pairs(c) ? 2 : 0;
}

// launch_groups: 1 launch before each lambda pass, 2 before each delta_p pass, 3 before xsph;
// with work lists 2 more before each lambda pass and one follower launch after
// each lambda and delta_p pass.
int group_launches(const StepConsts& c, int n, int niter) {
  // a small step: one launch before every pass (none before a lambda or xsph pass
  // with neither groups nor buckets, none before a delta_p pass without groups)
  if (is_small(c, n)) return n < kGroupCell ? (c.order ? niter : 0) : 2 * niter + 1;
  if (n < kGroupCell) return 0;
  return 3 * niter + 3 + (use_work_list(c, n) ? 4 * niter : 0);
}

}  // namespace pbf
