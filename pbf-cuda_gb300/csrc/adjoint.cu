// adjoint.cu — reverse pass of one step (pbf_backward): the vector-Jacobian
// product of the step with the neighbour sets and the clamp states of the
// forward held fixed.  The reference has no adjoint.
//
// Every pass is a gather over the same 27-cell windows as the forward (no
// atomics on per-particle results in the common case): a pair term that the
// forward adds to particle i's output also depends on particle j's inputs,
// and j gathers that transposed term from i when i lies in j's window too.
// Windows are centred on a particle's current cell but index the grid of the
// predicted positions, so a pair can be one-sided when a particle crossed a
// cell boundary during the step's iterations; each pair checks this
// (near_cell on the packed cells), and i scatters the terms that j cannot
// gather; they are summed exactly in any order (scatter_term, k_bwd_acc) and
// small kernels then fold them in, so the reverse pass is bitwise
// reproducible.
// Kernels:
//   W(q) = a (h^2 - q)^3,  W'(q) = -3a (h^2 - q)^2,  q = |r|^2
//   F(r) = phi(s) r,  phi = b (h - s)^2 / s,  s = |r|        (spiky gradient)
//   J(r) = dF/dr = phi I + (phi'(s) / s) r r^T,  phi' = -b (h - s)(h + s) / s^2
// Per iteration k (last to first), with X = X_k, lambda = lambda_k and the
// adjoint of X_{k+1} (k_bwd_window: delta_p 1, G_i and D_i of lambda 1, and the
// neighbour lists; k_bwd_delta_p: delta_p 2; k_bwd_fix_lambda: the rest of
// lambda 1; k_bwd_lambda: lambda 2):
//   delta_p 1: u = X + clamp(P / pho0), X_{k+1} = box(u): the clamps pass the
//              adjoint through where inactive, the wall takes it where active;
//              Pbar = ubar masked by the MAX_DP clamp / pho0
//   delta_p 2: lambdabar_i = sum_j F.(Pbar_i - Pbar_j)
//              xbar_i += sum_j (lambda_i + lambda_j + s_ij) J (Pbar_i - Pbar_j)
//                              + ds/dr (F.(Pbar_i - Pbar_j))
//   lambda 1:  Cbar = -lambdabar / D, Sbar = -lambdabar lambda / D (D = S + eps),
//              rhobar_tot = rhobar (last iteration, from XSPH) + Cbar / pho0
//   lambda 2:  xbar_i += sum_j 2 W'(q) r (rhobar_i + rhobar_j)
//                              + J (a_ij - a_ji) / pho0,  a_ij = 2 Sbar_i (g_ij + G_i)
// XSPH (nv_i = v_i + c sum_j (v_j - v_i) w_ij, w = 2 W / (rho_i + rho_j)):
//   vbar_i = nvbar_i + c sum_j w_ij (nvbar_j - nvbar_i)
//   xbar_i += sum_j c (nvbar_i - nvbar_j).(v_j - v_i) 2 W' / (rho_i + rho_j) 2 r
//   rhobar_i = sum_j c (nvbar_i - nvbar_j).(v_j - v_i) (-2 W / (rho_i + rho_j)^2)
#include <climits>

#include <cooperative_groups.h>

#include "pbf_internal.cuh"

namespace pbf {

namespace {

constexpr int kThreads = 128;
// Blocks, per block of the dense passes' grid, that take the particles without a
// list of a one-lane step: 8 per SM, what their registers allow (4 per SM: a
// crowded scene of 262,144 particles 30.5 ms, 8: 26.0, 20: 25.5, but 2% of a
// step without such particles).
constexpr int kLongBlocks = 2;
// Below this many particles a warp shares each particle (see lane_sum).  From
// 41,000 particles on one lane each is as fast or faster at rest (125,000: a
// gradient 1,333 us against 1,860), but loses where particles pile up (110,592,
// an eighth of them on 40 points: a reverse pass 4.5 ms against 2.0).
constexpr int kWarpPerParticleBelow = 131072;
// Lanes that split one particle's window in the reverse kernels of steps
// under kWarpPerParticleBelow particles: BackwardArgs::lanes (8, 16 or 32;
// pbf_tuning's bwd_lanes), 32 by default.  Few lanes suit windows of a few
// hundred candidates (less reduction per particle); many lanes suit piled-up
// states, where a handful of particles hold windows of thousands.

__device__ __forceinline__ void column_run(const SceneGeom& g, const uint32_t* __restrict__ cs,
                                           int n, int x, int y, int z, int& s, int& e) {
  const int zlo = max(z - 1, 0), zhi = min(z + 1, g.dims[2] - 1);
  const int base = g.cell_base + (x * g.dims[1] + y) * g.dims[2];
  s = (int)__ldg(cs + base + zlo);
  e = max(min((int)__ldg(cs + base + zhi + 1), n), s);
}

// f(j) for every candidate of the window of cell q, in order; with stride L,
// lane `lane` takes every L-th candidate of each run.
template <class F>
__device__ __forceinline__ void for_window(const SceneGeom& g, const uint32_t* __restrict__ cs,
                                           int n, int3 q, F&& f, int lane = 0, int stride = 1) {
  for (int dx = -1; dx <= 1; ++dx) {
    const int x = q.x + dx;
    if (x < 0 || x >= g.dims[0]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = q.y + dy;
      if (y < 0 || y >= g.dims[1]) continue;
      int s, e;
      column_run(g, cs, n, x, y, q.z, s, e);
      for (int j = s + lane; j < e; j += stride) f(j);
    }
  }
}

struct Vec {
  float x, y, z;
};
__device__ __forceinline__ Vec vsub(float4 a, float4 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float vdot(Vec a, Vec b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ __forceinline__ float dpoly6(const StepConsts& c, float q) {
  const float d = c.h2 - q;
  return -3.f * c.poly6_coef * d * d;
}

__device__ __forceinline__ float4 ld4(const float4* p, int i) { return __ldg(p + i); }

// Cells packed 21 bits per axis (grid dimensions are far below 2^21).
__device__ __forceinline__ unsigned long long pack_cell(int3 q) {
  return ((unsigned long long)q.x << 42) | ((unsigned long long)q.y << 21) | (unsigned long long)q.z;
}

// True when the cells differ by at most one along every axis, i.e. when a
// window centred on one contains the other.  All axes at once: 1 + a - b is 0, 1
// or 2 in every field, and the lowest field that is not shows it (no borrow
// reached it from below).
__device__ __forceinline__ bool near_cell(unsigned long long a, unsigned long long b) {
  constexpr unsigned long long kOnes = (1ull << 42) | (1ull << 21) | 1ull;
  const unsigned long long d = a + kOnes - b;
  return ((d & ~(3ull * kOnes)) | (d & (d >> 1) & kOnes)) == 0ull;
}

__device__ __forceinline__ void atomic_add3(float4* p, float x, float y, float z) {
  atomicAdd(&p->x, x);
  atomicAdd(&p->y, y);
  atomicAdd(&p->z, z);
}

// ---- exact scattered sums ------------------------------------------------------------
//
// A term that particle i cannot leave for j to gather is scattered to j.  Float
// atomics would add the terms in arrival order, so the result would change
// from run to run in its last bits; instead every term is listed (any order),
// each target keeps its term count and its largest finite |term| per component
// (integer atomics), k_bwd_acc then adds every listed term as a 64-bit integer
// scaled by 2^sh, sh = 62 - e - bits(count) with the largest |term| < 2^e (so
// no sum can overflow; integer sums do not depend on the order), and the fold
// converts back.  Each term is rounded to 2^-sh, at most 2^-62 of the target's
// largest term times its count: far below float rounding.  Non-finite terms
// are tracked per component (NaN, +inf, -inf) and give the IEEE sum's NaN or
// infinity.  Terms beyond the list's capacity go to fix / fixv with float
// atomics (results then correct but not bitwise reproducible; sc_ctr[1]
// counts them).

__device__ __forceinline__ int scale_shift(unsigned maxbits, unsigned cnt) {
  int e = 0;
  const float mx = __uint_as_float(maxbits);
  if (mx > 0.f) frexpf(mx, &e);  // mx < 2^e
  return 62 - e - (32 - __clz(cnt));
}

__device__ __forceinline__ void note_term(const BackwardArgs& a, int comp, int j, float v) {
  if (isfinite(v)) {
    if (v != 0.f) atomicMax(&a.sc_max[comp * a.sc_stride + j], __float_as_uint(fabsf(v)));
  } else {
    const unsigned bit = isnan(v) ? 1u : (v > 0.f ? 2u : 4u);
    atomicOr(&a.sc_nonfin[j], bit << (3 * comp));
  }
}

// Scatters (x, y, z, w) to target j: kind 0 (fix: position adjoints xyz and
// lambda / rho adjoint w) or kind 1 (fixv: velocity adjoints xyz).
__device__ __forceinline__ void scatter_term(const BackwardArgs& a, int kind, int j, float x, float y, float z,
                                             float w) {
  const unsigned slot = atomicAdd(&a.sc_ctr[a.sc_list], 1u);
  if (slot >= (unsigned)a.sc_cap) {
    atomicAdd(&a.sc_ctr[1], 1u);
    float4* f = kind == 0 ? a.fix : a.fixv;
    atomic_add3(f + j, x, y, z);
    if (kind == 0) atomicAdd(&f[j].w, w);
    return;
  }
  a.sc_key[slot] = make_int2(j, kind);
  a.sc_val[slot] = make_float4(x, y, z, w);
  atomicAdd(&a.sc_cnt[kind * a.sc_stride + j], 1u);
  const int base = kind == 0 ? 0 : 4;
  note_term(a, base, j, x);
  note_term(a, base + 1, j, y);
  note_term(a, base + 2, j, z);
  if (kind == 0) note_term(a, 3, j, w);
}

// Sums the wall adjoints of `blocks` blocks into g_lim[6] (accumulating) in a
// fixed order: thread t adds the parts of blocks t, t + kWallThreads, ... in
// turn, then the threads' sums are added pairwise in a fixed tree.
constexpr int kWallThreads = 256;
__device__ __forceinline__ void sum_walls(const float* __restrict__ part, int blocks, float* __restrict__ g_lim) {
  __shared__ float s[6][kWallThreads];
  float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int b = threadIdx.x; b < blocks; b += kWallThreads)
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] += part[b * 6 + k];
#pragma unroll
  for (int k = 0; k < 6; ++k) s[k][threadIdx.x] = acc[k];
  __syncthreads();
  for (int w = kWallThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
#pragma unroll
      for (int k = 0; k < 6; ++k) s[k][threadIdx.x] += s[k][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 6) g_lim[threadIdx.x] += s[threadIdx.x][0];
}

// Adds every listed term into its target's fixed-point sums (grid-stride), and
// empties the other list (the last one folded: two lists take turns, so no
// kernel reads a length that another block resets).  wall_blocks > 0: the last
// block sums that many blocks' wall adjoints instead.
__global__ void __launch_bounds__(kWallThreads) k_bwd_acc(BackwardArgs a, int wall_blocks, float* __restrict__ g_lim) {
  unsigned workers = gridDim.x;
  if (wall_blocks > 0) {
    if (blockIdx.x == --workers) {
      sum_walls(a.wall_part, wall_blocks, g_lim);
      return;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) a.sc_ctr[a.sc_list ^ 2] = 0u;
  const unsigned listed = min(a.sc_ctr[a.sc_list], (unsigned)a.sc_cap);
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < listed; e += workers * blockDim.x) {
    const int2 key = a.sc_key[e];
    const float4 v = a.sc_val[e];
    const int j = key.x, kind = key.y, base = kind == 0 ? 0 : 4, comps = kind == 0 ? 4 : 3;
    const unsigned cnt = a.sc_cnt[kind * a.sc_stride + j];
    const float vs[4] = {v.x, v.y, v.z, v.w};
    for (int c = 0; c < comps; ++c) {
      if (!isfinite(vs[c]) || vs[c] == 0.f) continue;
      const int comp = base + c;
      const int sh = scale_shift(a.sc_max[comp * a.sc_stride + j], cnt);
      const long long q = __double2ll_rn(ldexp((double)vs[c], sh));  // |q| < 2^62 / cnt
      atomicAdd(&a.sc_acc[comp * a.sc_stride + j], (unsigned long long)q);
    }
  }
}

// The exact sum of component `comp` of target j's listed terms, with its
// scratch set back to zero.
__device__ __forceinline__ float take_sum(const BackwardArgs& a, int comp, int j, unsigned cnt, unsigned nonfin) {
  const size_t k = (size_t)comp * a.sc_stride + j;
  const unsigned bits = (nonfin >> (3 * comp)) & 7u;
  const unsigned long long acc = a.sc_acc[k];
  const unsigned mx = a.sc_max[k];
  a.sc_acc[k] = 0ull;
  a.sc_max[k] = 0u;
  if (bits) {
    if ((bits & 1u) || (bits & 6u) == 6u) return __int_as_float(0x7fffffff);
    return (bits & 2u) ? __int_as_float(0x7f800000) : __int_as_float((int)0xff800000);
  }
  if (cnt == 0u || acc == 0ull) return 0.f;
  return (float)ldexp((double)(long long)acc, -scale_shift(mx, cnt));  // (few targets have terms)
}

// Target i's scattered sums of `kind` (xyz, and w for fix), its scratch
// cleared, plus what overflowed into fix / fixv (also cleared).  `listed`: the
// terms listed for all targets (0: nothing to read); false when none are i's.
__device__ __forceinline__ bool take_scattered(const BackwardArgs& a, int kind, int i, unsigned listed, float4& s) {
  s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (listed == 0u) return false;
  const unsigned cnt = a.sc_cnt[kind * a.sc_stride + i];
  if (cnt != 0u) {
    a.sc_cnt[kind * a.sc_stride + i] = 0u;
    const unsigned nonfin = a.sc_nonfin[i];
    const int base = kind == 0 ? 0 : 4;
    s.x = take_sum(a, base, i, cnt, nonfin);
    s.y = take_sum(a, base + 1, i, cnt, nonfin);
    s.z = take_sum(a, base + 2, i, cnt, nonfin);
    if (kind == 0) s.w = take_sum(a, 3, i, cnt, nonfin);
  }
  if (listed > (unsigned)a.sc_cap) {
    float4* f = kind == 0 ? a.fix : a.fixv;
    const float4 o = f[i];
    f[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    s = make_float4(s.x + o.x, s.y + o.y, s.z + o.z, kind == 0 ? s.w + o.w : 0.f);
    return true;
  }
  return cnt != 0u;
}

// After a fold: the target's non-finite bits of the folded kind are clear.
__device__ __forceinline__ void clear_nonfin(const BackwardArgs& a, int i, unsigned mask) {
  const unsigned nf = a.sc_nonfin[i];
  if (nf & mask) a.sc_nonfin[i] = nf & ~mask;
}

// L lanes share one particle (L = 1, or BackwardArgs::lanes for small steps,
// where one thread per particle would leave most SMs idle): its lanes split
// the window and add their sums in a fixed tree, so lane 0 holds the result.
template <int L>
__device__ __forceinline__ float lane_sum(float v) {
  if constexpr (L > 1) {
    // the L lanes of one particle are an aligned group of the warp (L divides
    // 32 and the blocks hold whole warps); they return together, so only the
    // group takes part: other groups of a warp may have returned already
    const unsigned lane = threadIdx.x & 31u;
    const unsigned mask = L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(unsigned)(L - 1));
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_down_sync(mask, v, o, L);
  }
  return v;
}

// phi(s) and phi'(s) / s of the spiky gradient F = phi r (|r| = s, q = s^2).  h - s
// takes s from a Newton step: near the cutoff s's own rounding would be most of
// phi's error (relative error over 0 < s < 0.95 h, in FP32 against FP64: phi 0.7e-7
// rms, phi' / s 1.0e-7; with a square root and two divisions 2.1e-7 and 1.6e-7).
__device__ __forceinline__ void spiky_parts(const StepConsts& c, float q, float& phi, float& k) {
  const float is = __frsqrt_rn(q), s = q * is;
  const float d = fmaf(-0.5f * is, fmaf(-s, s, q), c.h - s);
  phi = c.spiky_coef * d * d * is;
  k = -c.spiky_coef * d * (c.h + s) * is * is * is;
}

// ---- neighbour lists -------------------------------------------------------------------
//
// The window of a particle holds 216 candidates on average at rest and 33
// neighbours.  One kernel per iteration tests the candidates and lists the
// neighbours (the test the same as the lambda sums'), and all four sums of the
// iteration run over the list: lanes then stay together, and a sum gathers only
// what it needs.  A particle with more than kHitCap neighbours has no list
// (length -1): its sums walk the window, as every sum of every particle did
// before (with one lane per particle, a warp each: a crowded scene of 262,144
// particles 31.9 -> 26.0 ms).  Reverse pass of 262,144 particles at rest, 4
// iterations: 2,906 -> 1,060 us; of 15,625 (32 lanes per particle): 559 -> 231.
// Bounds: k_bwd_window (107 us a pass of 262,144 particles) issues instructions (64% of
// the slots: 85 million, three quarters of them tests and list entries), the
// sums over the lists wait for their gathers (47% of the slots).

// Entry k of particle i: one thread per particle interleaves the particles'
// lists (a warp reads entry k of its particles in one line), lanes of one
// particle read its list along.
template <int L>
__device__ __forceinline__ uint32_t* hit_list(const BackwardArgs& a, int i) {
  return a.hits + (L == 1 ? (size_t)i : (size_t)i * kHitCap);
}
template <int L>
__device__ __forceinline__ size_t hit_step(const BackwardArgs& a) {
  return L == 1 ? (size_t)a.hit_stride : 1;
}

constexpr uint32_t kOneSided = 0x80000000u;  // list entry: j cannot gather i's terms

// The lanes of particle i's group (all of a group's lanes run together).
template <int L>
__device__ __forceinline__ unsigned group_mask() {
  const unsigned lane = threadIdx.x & 31u;
  return L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(unsigned)(L - 1));
}

// Lists the candidates of particle i's window that lie within h of xi (or whose
// distance is NaN), itself among them, and returns their number, or -1 when they
// do not fit.
template <int L>
__device__ __forceinline__ int list_hits(const BackwardArgs& a, const float4* __restrict__ X, float4 xi, int i,
                                         int lane) {
  if (!a.hits) return -1;
  const StepConsts& c = a.c;
  const SceneGeom g = geom_of(c, a.G, i);
  const int3 q = cell_of(c, g, xi);
  uint32_t* list = hit_list<L>(a, i);
  int cnt = 0;
  const auto is_hit = [&](float4 xj) {
    const float r2 = dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
    return !(r2 >= c.h2);
  };
  if constexpr (L == 1) {
    // four candidates' loads in flight at a time, and room for four more entries
    // looked at once for them (so that a list holds kHitCap - 3 at least).  A full
    // list ends the innermost loop only: a lane that leaves all three at once may
    // reach the block's barriers after its warp was counted there (see solver.cu's
    // window_flagged)
    const size_t step = hit_step<L>(a);
    bool full = false;
    for (int dx = -1; dx <= 1; ++dx) {
      const int x = q.x + dx;
      if (x < 0 || x >= g.dims[0]) continue;
      for (int dy = -1; dy <= 1; ++dy) {
        const int y = q.y + dy;
        if (y < 0 || y >= g.dims[1]) continue;
        int s, e;
        column_run(g, a.cs, a.n, x, y, q.z, s, e);
        for (int j = s; j < e && !full; j += 4) {
          float4 xj[4];
          if (j + 4 <= a.n) {
#pragma unroll
            for (int u = 0; u < 4; ++u) xj[u] = ld4(X + j, u);
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) xj[u] = ld4(X, min(j + u, a.n - 1));
          }
          full = cnt > kHitCap - 4;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (!full && j + u < e && is_hit(xj[u])) {
              *list = (uint32_t)(j + u);
              list += step;
              ++cnt;
            }
          }
        }
      }
    }
    if (full) cnt = kHitCap + 1;
  } else {
    // the lanes look up the nine columns side by side, and every column's first
    // L candidates are in flight before the first test
    constexpr int kPer = (9 + L - 1) / L;
    const unsigned mask = group_mask<L>(), below = mask & ((1u << (threadIdx.x & 31u)) - 1u);
    int s[kPer], e[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int col = lane + p * L, x = q.x + col / 3 - 1, y = q.y + col % 3 - 1;
      s[p] = e[p] = 0;
      if (col < 9 && x >= 0 && x < g.dims[0] && y >= 0 && y < g.dims[1])
        column_run(g, a.cs, a.n, x, y, q.z, s[p], e[p]);
    }
    const auto append = [&](int j, bool hit) {
      const unsigned b = __ballot_sync(mask, hit);
      const int at = cnt + __popc(b & below);
      if (hit && at < kHitCap) list[at] = (uint32_t)j;
      cnt += __popc(b & mask);
    };
    float4 first[9];
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      const int j = __shfl_sync(mask, s[col / L], col % L, L) + lane;
      if (j < __shfl_sync(mask, e[col / L], col % L, L)) first[col] = ld4(X, j);
      else first[col] = xi;
    }
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      const int from = __shfl_sync(mask, s[col / L], col % L, L), to = __shfl_sync(mask, e[col / L], col % L, L);
      if (from >= to) continue;
      append(from + lane, from + lane < to && is_hit(first[col]));
      for (int j = from + lane + L; j - lane < to; j += L) append(j, j < to && is_hit(ld4(X, min(j, to - 1))));
    }
    __syncwarp(mask);  // the lanes read each other's entries
  }
  return cnt <= kHitCap ? cnt : -1;
}

template <int N>
struct Sums {
  float v[N];
};

// visit(own(i), sums, j, one-sided, load(j), null) for lane `lane` of `stride`'s
// share of the candidates of particle i's window that list_hits would list.
template <int N, class Own, class Load, class Visit>
__device__ __forceinline__ void walk_window(const BackwardArgs& a, const float4* __restrict__ X, int i, int lane,
                                            int stride, Sums<N>& sums, Own&& own, Load&& load, Visit&& visit) {
  const auto self = own(i);
  const float4 x = ld4(X, i);
  const SceneGeom g = geom_of(a.c, a.G, i);
  const unsigned long long cell = a.gcell[i];
  for_window(g, a.cs, a.n, cell_of(a.c, g, x), [&](int j) {
    const float4 xj = ld4(X, j);
    if (dist2(x.x - xj.x, x.y - xj.y, x.z - xj.z) >= a.c.h2) return;
    visit(self, sums, j, !near_cell(cell, a.kcell[j]), load(j), (uint32_t*)nullptr);
  }, lane, stride);
}

// finish(i, sums) in one lane for every particle i, sums over its neighbours
// what visit(own(i), sums, j, one-sided, load(j), list entry) adds: those of its
// list (the next one's loads in flight).  cnt: the list's length, or negative
// without one; with several lanes per particle they then walk the window, with
// one a warp of finish_long's does.
template <int L, int N, class Own, class Load, class Visit, class Finish>
__device__ __forceinline__ void finish_listed(const BackwardArgs& a, const float4* __restrict__ X, int i, int lane,
                                              int cnt, Own&& own, Load&& load, Visit&& visit, Finish&& finish) {
  if (L == 1 && cnt < 0) return;
  Sums<N> acc = {};
  if (lane < cnt) {
    const auto self = own(i);
    uint32_t* list = hit_list<L>(a, i);
    const size_t step = hit_step<L>(a);
    uint32_t e = list[lane * step];
    auto d = load((int)(e & ~kOneSided));
    for (int k = lane; k < cnt; k += L) {
      uint32_t en = e;
      auto dn = d;
      if (k + L < cnt) {
        en = list[(size_t)(k + L) * step];
        dn = load((int)(en & ~kOneSided));
      }
      visit(self, acc, (int)(e & ~kOneSided), (e & kOneSided) != 0u, d, list + (size_t)k * step);
      e = en;
      d = dn;
    }
  }
  if constexpr (L > 1) {
    if (cnt < 0) walk_window(a, X, i, lane, L, acc, own, load, visit);
#pragma unroll
    for (int k = 0; k < N; ++k) acc.v[k] = lane_sum<L>(acc.v[k]);
  }
  if (lane == 0) finish(i, acc);
}

// The same for the particles without a list of a one-lane step, a warp each.
// They come in runs (a crowded cell's particles), so warp w of W takes particles
// w, w + W, ...
template <int N, class Own, class Load, class Visit, class Finish>
__device__ __forceinline__ void finish_long(const BackwardArgs& a, const float4* __restrict__ X, int blocks,
                                            Own&& own, Load&& load, Visit&& visit, Finish&& finish) {
  const int lane = threadIdx.x & 31;
  const int W = blocks * (kThreads / 32), w = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  for (long long base = w; base < a.n; base += 32ll * W) {
    const long long i = base + (long long)lane * W;
    for (unsigned m = __ballot_sync(0xffffffffu, i < a.n && a.hit_n[i] < 0); m != 0u; m &= m - 1u) {
      const int of = (int)(base + (long long)(__ffs(m) - 1) * W);
      Sums<N> acc = {};
      walk_window(a, X, of, lane, 32, acc, own, load, visit);
#pragma unroll
      for (int k = 0; k < N; ++k) acc.v[k] = lane_sum<32>(acc.v[k]);
      if (lane == 0) finish(of, acc);
    }
  }
}

struct Two {
  float4 x, b;
};

// The packed cells of the grid's positions and of the final ones, the velocities
// v = (X_K - X0) / dt with rho, and empty lists of scattered terms.
__global__ void __launch_bounds__(256)
k_bwd_start(BackwardArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 2) a.sc_ctr[2 * i] = 0u;
  if (i >= a.n) return;
  const SceneGeom g = geom_of(a.c, a.G, i);
  const float4 x = ld4(a.XK, i), x0 = ld4(a.xs, i);
  a.gcell[i] = pack_cell(cell_of(a.c, g, ld4(a.X0, i)));
  a.kcell[i] = pack_cell(cell_of(a.c, g, x));
  a.pbar[i] = make_float4((x.x - x0.x) * a.c.inv_dt, (x.y - x0.y) * a.c.inv_dt, (x.z - x0.z) * a.c.inv_dt, a.rho[i]);
}

// ---- XSPH and the velocity update --------------------------------------------------

// kLong: the particles without a list of a one-lane step (after the others).
template <int L, bool kLong>
__global__ void __launch_bounds__(kThreads)
k_bwd_xsph(BackwardArgs a) {
  const StepConsts& c = a.c;
  struct Own {
    float4 x, v, g;
    unsigned long long cell;
    int i;
  };
  const auto own = [&](int k) { return Own{ld4(a.XK, k), ld4(a.pbar, k), ld4(a.g_nvel, k), a.gcell[k], k}; };
  const auto load = [&](int j) { return Two{ld4(a.XK, j), ld4(a.pbar, j)}; };
  const auto visit = [&](const Own& o, Sums<7>& s, int j, bool, const Two& t, uint32_t*) {
    const Vec r = vsub(o.x, t.x);
    const float q = vdot(r, r);
    if (!(q < c.h2) || j == o.i) return;
    const Vec dv = vsub(t.b, o.v);
    const float den = o.v.w + t.b.w;            // rho_i + rho_j
    const float w = 2.f * poly6_inside(c, q) / den;
    const float dq = 4.f * dpoly6(c, q) / den;  // d w / d x_i per unit of r
    const float dr = -w / den;                  // d w / d rho
    // nv_i's term c w (v_j - v_i) and, when i is in j's window, nv_j's
    // c w (v_i - v_j): their adjoints on i's inputs, from nvbar_i - nvbar_j
    const bool both = near_cell(o.cell, a.kcell[j]);
    Vec gd = {o.g.x, o.g.y, o.g.z};
    if (both) gd = vsub(o.g, ld4(a.g_nvel, j));
    const float gv = c.c_xsph * vdot(gd, dv);
    const float cw = c.c_xsph * w;
    s.v[0] -= cw * gd.x;
    s.v[1] -= cw * gd.y;
    s.v[2] -= cw * gd.z;
    s.v[3] += gv * dq * r.x;
    s.v[4] += gv * dq * r.y;
    s.v[5] += gv * dq * r.z;
    s.v[6] += gv * dr;
    if (!both) {
      // j cannot gather nv_i's term: scatter its adjoint on j's inputs
      scatter_term(a, 1, j, cw * gd.x, cw * gd.y, cw * gd.z, 0.f);
      scatter_term(a, 0, j, -gv * dq * r.x, -gv * dq * r.y, -gv * dq * r.z, gv * dr);
    }
  };
  const auto finish = [&](int i, const Sums<7>& s) {
    const float4 gi = ld4(a.g_nvel, i), gp = ld4(a.g_npos, i);
    const Vec vb = {gi.x + s.v[0], gi.y + s.v[1], gi.z + s.v[2]};  // nv_i = v_i + ...: the identity part
    // v = (X_K - X0) / dt: the position adjoint of the step's output plus XSPH's
    a.gx[i] = make_float4(gp.x + s.v[3] + vb.x * c.inv_dt, gp.y + s.v[4] + vb.y * c.inv_dt,
                          gp.z + s.v[5] + vb.z * c.inv_dt, 0.f);
    a.gx0[i] = make_float4(-vb.x * c.inv_dt, -vb.y * c.inv_dt, -vb.z * c.inv_dt, 0.f);
    a.grho[i] = s.v[6];
  };
  if constexpr (kLong) {
    finish_long<7>(a, a.XK, gridDim.x, own, load, visit, finish);
  } else {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t / L, lane = t % L;
    if (i >= a.n) return;
    const int cnt = list_hits<L>(a, a.XK, ld4(a.XK, i), i, lane);
    if (lane == 0) a.hit_n[i] = cnt;
    finish_listed<L, 7>(a, a.XK, i, lane, cnt, own, load, visit, finish);
  }
}

// The packed cells of the positions the next iteration's kernels work on (null: none follow).
__device__ __forceinline__ void next_cells(const BackwardArgs& a, const float4* __restrict__ X, int i) {
  if (X) a.kcell[i] = pack_cell(cell_of(a.c, geom_of(a.c, a.G, i), ld4(X, i)));
}

// Folds the scattered XSPH adjoints in and clears their scratch.
__global__ void __launch_bounds__(256)
k_bwd_fix_xsph(BackwardArgs a, const float4* __restrict__ next) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  next_cells(a, next, i);
  const unsigned listed = a.sc_ctr[a.sc_list];
  float4 f, v;
  const bool any = take_scattered(a, 0, i, listed, f), anyv = take_scattered(a, 1, i, listed, v);
  if (!any && !anyv) return;
  clear_nonfin(a, i, 0x1fffffu);
  const float4 g = a.gx[i], g0 = a.gx0[i];
  const float t = a.c.inv_dt;
  a.gx[i] = make_float4(g.x + f.x + v.x * t, g.y + f.y + v.y * t, g.z + f.z + v.z * t, 0.f);
  a.gx0[i] = make_float4(g0.x - v.x * t, g0.y - v.y * t, g0.z - v.z * t, 0.f);
  a.grho[i] += f.w;
}

// Folds the lambda sums' scattered position adjoints into gx_next and clears
// their scratch.
__global__ void __launch_bounds__(256)
k_bwd_fix(BackwardArgs a, const float4* __restrict__ next) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  next_cells(a, next, i);
  float4 f;
  if (!take_scattered(a, 0, i, a.sc_ctr[a.sc_list], f)) return;
  clear_nonfin(a, i, 0xfffu);
  const float4 g = a.gx_next[i];
  a.gx_next[i] = make_float4(g.x + f.x, g.y + f.y, g.z + f.z, 0.f);
}

// ---- delta_p -----------------------------------------------------------------------

// Lists every particle's neighbours, recomputes P_i (the forward's sum) and the
// lambda sums (G_i and D_i), applies the clamps' transposes.  Writes Pbar,
// starts the X_k adjoint with ubar, and leaves this block's wall adjoints in
// wall_part[block][6] (ulim xyz, llim xyz).  kLong: as k_bwd_xsph's.
template <int L, bool kLong>
__global__ void __launch_bounds__(kThreads)
k_bwd_window(BackwardArgs a, const float4* __restrict__ X, const float* __restrict__ lam, float* __restrict__ wall_part) {
  const StepConsts& c = a.c;
  __shared__ float wall[6][kThreads / 32];
  struct Own {
    float4 x;
    float lam;
    unsigned long long cell;
    int i;
  };
  struct Pair {
    float4 x;
    float lam;
    unsigned long long cell;
  };
  const auto own = [&](int k) { return Own{ld4(X, k), __ldg(lam + k), a.gcell[k], k}; };
  const auto load = [&](int j) { return Pair{ld4(X, j), __ldg(lam + j), a.kcell[j]}; };
  // P (0-2), G (3-5), sum of |g_ij|^2 (6)
  const auto visit = [&](const Own& o, Sums<7>& s, int j, bool, const Pair& t, uint32_t* entry) {
    if (entry && !near_cell(o.cell, t.cell)) *entry = (uint32_t)j | kOneSided;
    const float ex = o.x.x - t.x.x, ey = o.x.y - t.x.y, ez = o.x.z - t.x.z;
    const float r2 = dist2(ex, ey, ez);
    if (r2 >= c.h2 || r2 < c.keps2) return;
    const float ir = rsqrtf(r2);
    const float d = c.h - r2 * ir;
    const float sc = c.spiky_coef_rho0 * d * d * ir;
    s.v[3] += sc * ex;
    s.v[4] += sc * ey;
    s.v[5] += sc * ez;
    if (j != o.i) {
      const float corr = c.coef_corr * pow_corr(c, poly6_inside(c, r2));
      const float f = (o.lam + t.lam + corr) * (c.spiky_coef * d * d * ir);
      s.v[0] = fmaf(f, ex, s.v[0]);
      s.v[1] = fmaf(f, ey, s.v[1]);
      s.v[2] = fmaf(f, ez, s.v[2]);
      s.v[6] += dist2(sc * ex, sc * ey, sc * ez);
    }
  };
  float w6[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const auto finish = [&](int i, const Sums<7>& s) {
    const SceneGeom g = geom_of(c, a.G, i);
    const float4 xi = ld4(X, i), gn = ld4(a.gx, i);  // gx: the adjoint of X_{k+1}
    const float x[3] = {xi.x, xi.y, xi.z}, gin[3] = {gn.x, gn.y, gn.z};
    float ub[3], pb[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      const float dpa = s.v[ax] / c.pho0;
      const float u = x[ax] + fmaxf(fminf(dpa, c.max_dp), -c.max_dp);
      ub[ax] = gin[ax];
      if (u > g.hi[ax]) {
        w6[ax] += gin[ax];
        ub[ax] = 0.f;
      } else if (u < g.lo[ax]) {
        w6[3 + ax] += gin[ax];
        ub[ax] = 0.f;
      }
      pb[ax] = (dpa < c.max_dp && dpa > -c.max_dp) ? ub[ax] / c.pho0 : 0.f;
    }
    a.pbar[i] = make_float4(pb[0], pb[1], pb[2], lam[i]);
    a.gx_next[i] = make_float4(ub[0], ub[1], ub[2], 0.f);
    a.gs[i] = make_float4(s.v[3], s.v[4], s.v[5], s.v[6] + dist2(s.v[3], s.v[4], s.v[5]) + c.lambda_eps);
  };
  if constexpr (kLong) {
    finish_long<7>(a, X, gridDim.x, own, load, visit, finish);
  } else {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = tid / L, lane = tid % L;
    if (i < a.n) {
      const int cnt = list_hits<L>(a, X, ld4(X, i), i, lane);
      if (lane == 0) a.hit_n[i] = cnt;
      finish_listed<L, 7>(a, X, i, lane, cnt, own, load, visit, finish);
    }
  }
  // this block's wall adjoints, added in a fixed tree (mostly all zero)
  const bool some = w6[0] != 0.f || w6[1] != 0.f || w6[2] != 0.f || w6[3] != 0.f || w6[4] != 0.f || w6[5] != 0.f;
  const bool any = __syncthreads_or(some) != 0;
  if (any) {
    for (int k = 0; k < 6; ++k) {
      float v = w6[k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) wall[k][threadIdx.x >> 5] = v;
    }
    __syncthreads();
  }
  if (threadIdx.x < 6) {
    float sum = 0.f;
    if (any)
      for (int k = 0; k < kThreads / 32; ++k) sum += wall[threadIdx.x][k];
    wall_part[blockIdx.x * 6 + threadIdx.x] = sum;
  }
}

// long_blocks: with one lane per particle, the first blocks take the particles
// without a list.
template <int L>
__global__ void __launch_bounds__(kThreads)
k_bwd_delta_p(BackwardArgs a, const float4* __restrict__ X, int long_blocks) {
  const StepConsts& c = a.c;
  struct Own {
    float4 x, p;
    int i;
  };
  const auto own = [&](int k) { return Own{ld4(X, k), ld4(a.pbar, k), k}; };
  const auto load = [&](int j) { return Two{ld4(X, j), ld4(a.pbar, j)}; };
  const auto visit = [&](const Own& o, Sums<4>& s, int j, bool one_sided, const Two& t, uint32_t*) {
    const Vec r = vsub(o.x, t.x);
    const float q = vdot(r, r);
    if (!(q < c.h2) || q < c.keps2 || j == o.i) return;
    float phi, k;
    spiky_parts(c, q, phi, k);
    const float wq = poly6_inside(c, q);
    const float lsum = o.p.w + t.b.w + c.coef_corr * pow_corr(c, wq);
    const float dsdq = c.npow == 4 ? 4.f * c.coef_corr * wq * wq * wq * dpoly6(c, q)
                                   : c.coef_corr * c.n_corr * powf(wq, c.n_corr - 1.f) * dpoly6(c, q);
    // P_i's term (lambda_i + lambda_j + s_ij) F(r_ij) and, when i is in j's
    // window, P_j's (F and r change sign, J does not): their adjoints on
    // lambda_i and x_i, from d = Pbar_i - Pbar_j
    Vec d = {o.p.x, o.p.y, o.p.z};
    if (!one_sided) d = vsub(o.p, t.b);
    const float rd = vdot(r, d), fd = phi * rd;
    const float u = lsum * phi, v = lsum * k * rd + 2.f * dsdq * fd;
    const Vec x = {u * d.x + v * r.x, u * d.y + v * r.y, u * d.z + v * r.z};
    s.v[0] += x.x;
    s.v[1] += x.y;
    s.v[2] += x.z;
    s.v[3] += fd;
    // j cannot gather P_i's term: scatter its adjoint on lambda_j and x_j
    if (one_sided) scatter_term(a, 0, j, -x.x, -x.y, -x.z, fd);
  };
  const auto finish = [&](int i, const Sums<4>& s) {
    const float4 u = ld4(a.gx_next, i);
    a.gx_next[i] = make_float4(u.x + s.v[0], u.y + s.v[1], u.z + s.v[2], 0.f);
    a.lbar[i] = s.v[3];
  };
  if (L == 1 && (int)blockIdx.x < long_blocks) {
    finish_long<4>(a, X, long_blocks, own, load, visit, finish);
    return;
  }
  const int tid = ((int)blockIdx.x - long_blocks) * kThreads + threadIdx.x;
  const int i = tid / L, lane = tid % L;
  if (i < a.n) finish_listed<L, 4>(a, X, i, lane, a.hit_n[i], own, load, visit, finish);
}

// ---- lambda ------------------------------------------------------------------------

// Folds the delta_p sums' scattered adjoints in and clears their scratch; then
// the constraint's adjoints: Sbar_i beside 2 Sbar_i G_i, rho's beside X_i.
__global__ void __launch_bounds__(256)
k_bwd_fix_lambda(BackwardArgs a, const float4* __restrict__ X, const float* __restrict__ lam, int last) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  float lb = a.lbar[i];
  float4 f;
  if (take_scattered(a, 0, i, a.sc_ctr[a.sc_list], f)) {
    clear_nonfin(a, i, 0xfffu);
    const float4 g = a.gx_next[i];
    a.gx_next[i] = make_float4(g.x + f.x, g.y + f.y, g.z + f.z, 0.f);
    lb += f.w;
  }
  const float4 g = a.gs[i], x = ld4(X, i);
  const float cbar = -lb / g.w;
  const float sbar = -lb * lam[i] / g.w;
  const float s2 = 2.f * sbar;
  a.gs[i] = make_float4(s2 * g.x, s2 * g.y, s2 * g.z, s2);
  a.pbar[i] = make_float4(x.x, x.y, x.z, (last ? a.grho[i] : 0.f) + cbar / a.c.pho0);
}

template <int L>
__global__ void __launch_bounds__(kThreads)
k_bwd_lambda(BackwardArgs a, int long_blocks) {
  const StepConsts& c = a.c;
  struct Own {
    float4 x, g;
    int i;
  };
  const auto own = [&](int k) { return Own{ld4(a.pbar, k), ld4(a.gs, k), k}; };
  const auto load = [&](int j) { return Two{ld4(a.pbar, j), ld4(a.gs, j)}; };
  const auto visit = [&](const Own& o, Sums<3>& s, int j, bool one_sided, const Two& t, uint32_t*) {
    const Vec r = vsub(o.x, t.x);
    const float q = vdot(r, r);
    if (!(q < c.h2) || j == o.i) return;
    // rho_i's term W(q) and, when i is in j's window, rho_j's: 2 W'(q) r times
    // the adjoints of rho on x_i, minus that on x_j
    const float wt = 2.f * dpoly6(c, q) * (one_sided ? o.x.w : o.x.w + t.x.w);
    Vec x = {wt * r.x, wt * r.y, wt * r.z};
    if (!(q < c.keps2)) {
      // S_i's terms |g_ij|^2 + the g_ij part of |G_i|^2, g_ij = F / pho0:
      // a_ij = 2 Sbar_i (g_ij + G_i); S_j's a_ji = 2 Sbar_j (-g_ij + G_j):
      // J (a_ij - a_ji) / pho0 on x_i, minus that on x_j
      float phi, k;
      spiky_parts(c, q, phi, k);
      Vec v = {o.g.x, o.g.y, o.g.z};
      float s2 = o.g.w;
      if (!one_sided) {
        v = vsub(o.g, t.b);
        s2 += t.b.w;
      }
      const float m = phi * c.inv_pho0, sp = s2 * m;
      v = {v.x + sp * r.x, v.y + sp * r.y, v.z + sp * r.z};
      const float n = k * vdot(r, v) * c.inv_pho0;
      x = {x.x + (m * v.x + n * r.x), x.y + (m * v.y + n * r.y), x.z + (m * v.z + n * r.z)};
    }
    s.v[0] += x.x;
    s.v[1] += x.y;
    s.v[2] += x.z;
    if (one_sided) scatter_term(a, 0, j, -x.x, -x.y, -x.z, 0.f);
  };
  const auto finish = [&](int i, const Sums<3>& s) {
    const float4 u = ld4(a.gx_next, i);
    a.gx_next[i] = make_float4(u.x + s.v[0], u.y + s.v[1], u.z + s.v[2], 0.f);
  };
  if (L == 1 && (int)blockIdx.x < long_blocks) {
    finish_long<3>(a, a.pbar, long_blocks, own, load, visit, finish);
    return;
  }
  const int tid = ((int)blockIdx.x - long_blocks) * kThreads + threadIdx.x;
  const int i = tid / L, lane = tid % L;
  if (i < a.n) finish_listed<L, 3>(a, a.pbar, i, lane, a.hit_n[i], own, load, visit, finish);
}

// ---- advection and the permutation ---------------------------------------------------

// x* = x + dt v + dt^2 g: adjoints of the (sorted) inputs, scattered back to
// the caller's input order through the sort permutation.
__global__ void __launch_bounds__(256)
k_bwd_out(BackwardArgs a, const uint32_t* __restrict__ perm, float4* __restrict__ g_pos,
          float4* __restrict__ g_vel) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < 2) a.sc_ctr[2 * k] = 0u;  // both lists, for the next call
  if (k >= a.n) return;
  const float4 gs = ld4(a.gx, k), g0 = ld4(a.gx0, k);
  const uint32_t p = min(perm[k], (uint32_t)(a.n - 1));
  g_pos[p] = make_float4(gs.x + g0.x, gs.y + g0.y, gs.z + g0.z, 0.f);
  g_vel[p] = make_float4(a.c.dt * gs.x, a.c.dt * gs.y, a.c.dt * gs.z, 0.f);
}

// ---- density grid ---------------------------------------------------------------------

struct Lattice {
  float lo[3], step[3];
  int dims[3];
  float h, h2, coef;  // poly6 radius and coefficient
};

Lattice make_lattice(const float lo[3], const float hi[3], const int dims[3], float h) {
  Lattice L;
  for (int a = 0; a < 3; ++a) {
    L.lo[a] = lo[a];
    L.dims[a] = dims[a];
    L.step[a] = (hi[a] - lo[a]) / (float)dims[a];
  }
  L.h = h;
  L.h2 = h * h;
  L.coef = (float)(315.0 / (64.0 * kRefPi * (double)h * h * h * h * h * h * h * h * h));
  return L;
}

__device__ __forceinline__ float node_coord(const Lattice& L, int a, int k) {
  return L.lo[a] + ((float)k + 0.5f) * L.step[a];
}

// A block holds a brick of 4 x 8 x 8 nodes, one per thread (a warp: 2 x 4 x 4
// of them), and streams its share of the particles through two culls: a
// particle that no node of the brick can reach is dropped on load, the others
// are compacted in order into shared memory, and each warp drops those that
// none of its own 32 nodes can reach before its lanes visit the rest.  The
// nearest node's bound is computed with the node test's own operations, each
// monotonic in float arithmetic, so a cull never drops a particle that the
// node test would take.  A cluster of kGridSplit blocks shares a brick, each
// taking every kGridSplit-th batch of particles (they come in cell order, so
// contiguous parts would leave one block all of the brick's survivors); the
// blocks' sums are added in rank order through distributed shared memory (no
// scratch in global memory, and the same sum on every run).
//
// Bound by instruction issue: the culls cost ~20 instructions per particle and
// brick and ~15 per survivor and warp, against ~10 per particle and NODE when
// every node tested every particle (the earlier kernel).  A brick smaller than
// 256 nodes would stream the particles through more blocks (L2 reads), a
// larger one leaves its warps more survivors.  The kernel's time on GB300:
// 262,144 particles on 32^3 nodes 4,549 -> 127 us, 15,625 on 32 x 16 x 16
// 275 -> 25 us.
constexpr int kGridThreads = 256, kGridSplit = 8;
// A cluster shares a brick where there is at most one brick per SM; with more,
// whole blocks fill the chip, and streaming the particles through eight times the
// blocks costs more than it gains where they are few or spread over the lattice
// (15,625 particles: 128 bricks 17 us split, 48 whole; 512 bricks 52 and 37;
// 262,144 in an eighth of the lattice's box, whose bricks hold unequal work: 184
// and 733, 226 and 412, 1,024 bricks 398 and 330).
constexpr int kGridMaxBricks = 1 << 20;              // bricks in flight (the blocks loop over the rest)
constexpr int kGridUnroll = 4;                       // particles in flight per thread
constexpr int kGridBatch = kGridThreads * kGridUnroll;
constexpr int kGridWarps = kGridThreads / 32;
constexpr int kBrickX = 4, kBrickY = 8, kBrickZ = 8;  // nodes of a brick per axis
static_assert(kBrickX * kBrickY * kBrickZ == kGridThreads, "one node per thread");
static_assert(kGridWarps * kGridUnroll == 32, "one warp scans a batch's survivor counts");

// The interval per axis that the coordinates of nodes [k, k + count) span,
// clipped to the lattice.
struct NodeBox {
  float lo[3], hi[3];
};
__device__ __forceinline__ NodeBox node_box(const Lattice& L, unsigned kx, unsigned ky, unsigned kz, unsigned cx,
                                            unsigned cy, unsigned cz) {
  const unsigned k0[3] = {kx, ky, kz}, count[3] = {cx, cy, cz};
  NodeBox b;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = node_coord(L, a, (int)min(k0[a], L.dims[a] - 1u));
    b.hi[a] = node_coord(L, a, (int)min(k0[a] + count[a] - 1u, L.dims[a] - 1u));
  }
  return b;
}
// Whether x may lie within the radius of a node of the box.
__device__ __forceinline__ bool reaches(const NodeBox& b, float4 x, float h2) {
  const float ex = fmaxf(fmaxf(b.lo[0] - x.x, x.x - b.hi[0]), 0.f);
  const float ey = fmaxf(fmaxf(b.lo[1] - x.y, x.y - b.hi[1]), 0.f);
  const float ez = fmaxf(fmaxf(b.lo[2] - x.z, x.z - b.hi[2]), 0.f);
  return dist2(ex, ey, ez) < h2;
}

template <int kSplit>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kGridThreads)
k_density_grid(const float4* __restrict__ pos, int n, Lattice L, unsigned bricks, unsigned batch,
               float* __restrict__ grid) {
  namespace cg = cooperative_groups;
  __shared__ float4 keep[kGridBatch];
  __shared__ int counts[33];
  __shared__ float sums[kGridThreads];
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned part = cluster.block_rank();
  const unsigned by = ((unsigned)L.dims[1] + kBrickY - 1) / kBrickY, bz = ((unsigned)L.dims[2] + kBrickZ - 1) / kBrickZ;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (unsigned brick = blockIdx.x / kSplit; brick < bricks; brick += gridDim.x / kSplit) {
    const unsigned k0[3] = {brick / (by * bz) * kBrickX, brick / bz % by * kBrickY, brick % bz * kBrickZ};
    // a warp's 2 x 4 x 4 nodes, z fastest over the lanes
    const unsigned w0[3] = {k0[0] + (warp >> 2) * 2, k0[1] + ((warp >> 1) & 1) * 4, k0[2] + (warp & 1) * 4};
    const unsigned kx = w0[0] + (lane >> 4), ky = w0[1] + ((lane >> 2) & 3), kz = w0[2] + (lane & 3);
    const float px = node_coord(L, 0, (int)kx), py = node_coord(L, 1, (int)ky), pz = node_coord(L, 2, (int)kz);
    const NodeBox brick_box = node_box(L, k0[0], k0[1], k0[2], kBrickX, kBrickY, kBrickZ);
    const NodeBox warp_box = node_box(L, w0[0], w0[1], w0[2], 2, 4, 4);
    float d = 0.f;
    // unsigned: base passes 2^31 for the largest n
    for (unsigned base = part * batch; base < (unsigned)n; base += kSplit * batch) {
      float4 x[kGridUnroll];
      unsigned ballot[kGridUnroll], some = 0u;
      const unsigned end = min(base + batch, (unsigned)n);
#pragma unroll
      for (int u = 0; u < kGridUnroll; ++u) x[u] = __ldg(pos + min(base + u * kGridThreads + threadIdx.x, end - 1u));
#pragma unroll
      for (int u = 0; u < kGridUnroll; ++u) {
        const bool in = base + u * kGridThreads + threadIdx.x < end;
        ballot[u] = __ballot_sync(0xffffffffu, in && reaches(brick_box, x[u], L.h2));
        some |= ballot[u];
        if (lane == 0) counts[u * kGridWarps + warp] = __popc(ballot[u]);
      }
      if (!__syncthreads_or(some != 0u)) continue;  // no survivor: nobody reads counts
      if (warp == 0) {  // exclusive offsets of the batch's 32 (round, warp) groups
        const int v = counts[lane];
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, s, o);
          if (lane >= o) s += y;
        }
        counts[lane] = s - v;
        if (lane == 31) counts[32] = s;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kGridUnroll; ++u)
        if (ballot[u] >> lane & 1u) keep[counts[u * kGridWarps + warp] + __popc(ballot[u] & ((1u << lane) - 1u))] = x[u];
      const int m = counts[32];
      __syncthreads();
      for (int k = 0; k < m; k += 32) {
        unsigned todo = __ballot_sync(0xffffffffu, k + lane < m && reaches(warp_box, keep[min(k + lane, m - 1)], L.h2));
        while (todo) {
          const float4 p = keep[k + __ffs(todo) - 1];
          todo &= todo - 1u;
          const float q = dist2(p.x - px, p.y - py, p.z - pz);
          if (q < L.h2) {
            const float w = L.h2 - q;
            d += L.coef * w * w * w;
          }
        }
      }
      __syncthreads();  // the batch's readers are done with keep and counts
    }
    if (kSplit > 1) {
      sums[threadIdx.x] = d;
      cluster.sync();
      if (part == 0)
        for (int p = 1; p < kSplit; ++p) d += cluster.map_shared_rank(sums, p)[threadIdx.x];
    }
    if (part == 0 && kx < (unsigned)L.dims[0] && ky < (unsigned)L.dims[1] && kz < (unsigned)L.dims[2])
      grid[((size_t)kx * L.dims[1] + ky) * L.dims[2] + kz] = d;
    if (kSplit > 1) cluster.sync();  // the other blocks' sums stay in place until they are read
  }
}

// Per particle: the nodes within h (a box of lattice indices around it).
__global__ void __launch_bounds__(256)
k_density_grid_backward(const float4* __restrict__ pos, int n, Lattice L,
                        const float* __restrict__ g_grid, float4* __restrict__ g_pos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 x = pos[i];
  const float p[3] = {x.x, x.y, x.z};
  int klo[3], khi[3];
  for (int a = 0; a < 3; ++a) {
    klo[a] = max((int)floorf((p[a] - L.h - L.lo[a]) / L.step[a] - 0.5f), 0);
    khi[a] = min((int)ceilf((p[a] + L.h - L.lo[a]) / L.step[a] - 0.5f), L.dims[a] - 1);
  }
  float gx = 0.f, gy = 0.f, gz = 0.f;
  for (int a = klo[0]; a <= khi[0]; ++a)
    for (int b = klo[1]; b <= khi[1]; ++b)
      for (int cz = klo[2]; cz <= khi[2]; ++cz) {
        const float rx = x.x - node_coord(L, 0, a), ry = x.y - node_coord(L, 1, b),
                    rz = x.z - node_coord(L, 2, cz);
        const float q = dist2(rx, ry, rz);
        if (!(q < L.h2)) continue;
        const float w = L.h2 - q;
        const float gq = g_grid[(a * L.dims[1] + b) * L.dims[2] + cz] * (-3.f * L.coef * w * w) * 2.f;
        gx += gq * rx;
        gy += gq * ry;
        gz += gq * rz;
      }
  g_pos[i] = make_float4(gx, gy, gz, 0.f);
}

}  // namespace

cudaError_t density_grid(const float4* pos, int n, const float lo[3], const float hi[3],
                         const int dims[3], float h, float* grid, cudaStream_t stream) {
  const Lattice L = make_lattice(lo, hi, dims, h);
  const long long bricks = ((long long)dims[0] + kBrickX - 1) / kBrickX * (((long long)dims[1] + kBrickY - 1) / kBrickY) *
                           (((long long)dims[2] + kBrickZ - 1) / kBrickZ);
  const unsigned resident = (unsigned)min(bricks, (long long)kGridMaxBricks);
  // few particles: shorter batches, so that every block of a cluster has one (1,000
  // particles on 8^3 nodes: 41 us with whole batches)
  const unsigned batch = min((unsigned)kGridBatch, max(32u, ((unsigned)n / kGridSplit + 31u) / 32u * 32u));
  if (bricks <= device_sms())
    k_density_grid<kGridSplit><<<resident * kGridSplit, kGridThreads, 0, stream>>>(pos, n, L, (unsigned)bricks, batch,
                                                                                     grid);
  else
    k_density_grid<1><<<resident, kGridThreads, 0, stream>>>(pos, n, L, (unsigned)bricks, kGridBatch, grid);
  return cudaGetLastError();
}

cudaError_t density_grid_backward(const float4* pos, int n, const float lo[3], const float hi[3],
                                  const int dims[3], float h, const float* g_grid, float4* g_pos,
                                  cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const Lattice L = make_lattice(lo, hi, dims, h);
  k_density_grid_backward<<<(n + 255) / 256, 256, 0, stream>>>(pos, n, L, g_grid, g_pos);
  return cudaGetLastError();
}

template <int L>
cudaError_t run_backward(BackwardArgs a, const BackwardTape& t, const uint32_t* perm, void* g_pos,
                         void* g_vel, float* g_lim, cudaStream_t stream) {
  const int blocks = (int)(((long long)a.n * L + kThreads - 1) / kThreads);
  const int blocks256 = (a.n + 255) / 256;
  const int acc_blocks = a.c.dense_grid;
  const int K = t.niter;
  const int longs = L == 1 ? kLongBlocks * acc_blocks : 0;  // blocks for the particles without a list
  k_bwd_xsph<L, false><<<blocks, kThreads, 0, stream>>>(a);
  if constexpr (L == 1) k_bwd_xsph<1, true><<<longs, kThreads, 0, stream>>>(a);
  k_bwd_acc<<<acc_blocks, kWallThreads, 0, stream>>>(a, 0, g_lim);
  k_bwd_fix_xsph<<<blocks256, 256, 0, stream>>>(a, K > 0 ? t.X[K - 1] : nullptr);
  a.sc_list ^= 2;
  for (int k = K - 1; k >= 0; --k) {
    const float4* X = t.X[k];
    const float* lam = t.lambda[k];
    k_bwd_window<L, false><<<blocks, kThreads, 0, stream>>>(a, X, lam, a.wall_part);
    if constexpr (L == 1) k_bwd_window<1, true><<<longs, kThreads, 0, stream>>>(a, X, lam, a.wall_part + 6 * blocks);
    k_bwd_delta_p<L><<<longs + blocks, kThreads, 0, stream>>>(a, X, longs);
    k_bwd_acc<<<acc_blocks + 1, kWallThreads, 0, stream>>>(a, blocks + longs, g_lim);
    k_bwd_fix_lambda<<<blocks256, 256, 0, stream>>>(a, X, lam, k == K - 1);
    a.sc_list ^= 2;
    k_bwd_lambda<L><<<longs + blocks, kThreads, 0, stream>>>(a, longs);
    k_bwd_acc<<<acc_blocks, kWallThreads, 0, stream>>>(a, 0, g_lim);
    k_bwd_fix<<<blocks256, 256, 0, stream>>>(a, k > 0 ? t.X[k - 1] : nullptr);
    a.sc_list ^= 2;
    // the adjoint of X_k becomes the input of the next (earlier) iteration
    float4* tmp = a.gx;
    a.gx = a.gx_next;
    a.gx_next = tmp;
  }
  k_bwd_out<<<(a.n + 255) / 256, 256, 0, stream>>>(a, perm, (float4*)g_pos, (float4*)g_vel);
  return cudaGetLastError();
}

cudaError_t backward(const BackwardArgs& args, const BackwardTape& t, const uint32_t* perm,
                     const void* g_npos, const void* g_nvel, void* g_pos, void* g_vel,
                     float* g_lim, cudaStream_t stream) {
  BackwardArgs a = args;
  a.g_npos = (const float4*)g_npos;
  a.g_nvel = (const float4*)g_nvel;
  cudaError_t e = cudaMemsetAsync(g_lim, 0, sizeof(float) * 6, stream);
  if (e != cudaSuccess) return e;
  a.XK = t.X[t.niter];
  a.X0 = t.X[0];
  const int blocks256 = (a.n + 255) / 256;
  k_bwd_start<<<blocks256, 256, 0, stream>>>(a);
  if (a.n < kWarpPerParticleBelow) {
    if (a.lanes == 8) return run_backward<8>(a, t, perm, g_pos, g_vel, g_lim, stream);
    if (a.lanes == 16) return run_backward<16>(a, t, perm, g_pos, g_vel, g_lim, stream);
    return run_backward<32>(a, t, perm, g_pos, g_vel, g_lim, stream);
  }
  return run_backward<1>(a, t, perm, g_pos, g_vel, g_lim, stream);
}

}  // namespace pbf
