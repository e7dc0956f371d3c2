// kernels_sweep.cuh -- triangular sweeps over subtree tasks (task_plan.hpp).
//
// A sweep does one multiply-add per factor element, so what it can reach is
// the bandwidth of one pass over the factors; a launch per level of the tree
// instead pays a chain of dependent memory round trips per level.  Here a
// team sweeps a whole subtree: the factors of the next front arrive by
// cp.async while the current one is solved, and everything that passes
// between the fronts of the task (solution rows, update vectors) stays in
// shared memory.  Teams, lanes and workers as in kernels_task.cuh.  The backward
// sweep U x = y stays with the level kernels: its order makes a front one
// serial chain, which gains nothing from a team (10,000 buses x 64: 227 us as
// tasks, 162 us by levels).  Measured, the factorization's tasks included:
// factorize + solve + transpose solve of 1,024 FP32 Jacobians of the 2,000-bus
// grid 1,740 -> 1,238 us; forward and backward through torch on 10,000 buses x
// 64 9.14 -> 5.28 ms.  The stages of one L sweep there
// (2,000 x 1,024 FP32): 15, 4 and 2 resident warps on an SM, 52, 20 and 13 % of
// the issue slots, DRAM at 12, 6 and 2 %: the chain of fronts, not bandwidth.
#pragma once

#include <type_traits>

#include "kernels_task.cuh"

namespace cupf_b200 {
namespace {

// Factor elements of one front in the order a sweep stages them.
enum SweepMode { kSweepL = 0, kSweepUT = 1, kSweepLT = 2 };

template <typename T, int V, int LS, int TW>
struct Sweeper {
  using Team = TaskTeam<T, V, LS, TW>;
  using P = Pack<T, V>;
  using R = Rows<T, Team::S>;
  static constexpr int S = Team::S;

  const SweepTaskArgs<T>& a;
  size_t col0;
  int tid, worker, s0;

  __device__ __forceinline__ P ld(const T* base, int e) const {
    return *reinterpret_cast<const P*>(base + e * S + s0);
  }
  __device__ __forceinline__ void st(T* base, int e, const P& v) const { *reinterpret_cast<P*>(base + e * S + s0) = v; }
  __device__ __forceinline__ void out(T* g, size_t e, const P& v) const {
    *reinterpret_cast<P*>(g + e * a.Bp + col0 + s0) = v;
  }
  // n consecutive elements of a [element][Bp] array into shared memory
  __device__ __forceinline__ void fetch(T* smem, const T* g, size_t e0, int n) const {
    constexpr int PP = R::kPieces;
    const size_t row = (size_t)a.Bp * sizeof(T);
    const unsigned char* src = reinterpret_cast<const unsigned char*>(g) + e0 * row + col0 * sizeof(T);
    unsigned char* dst = reinterpret_cast<unsigned char*>(smem);
    for (int i = tid; i < n * PP; i += Team::NT) {
      const int e = i / PP, piece = (i % PP) * R::kPiece;
      R::fetch(dst + e * R::kBytes + piece, src + (size_t)e * row + piece);
    }
  }
  // The front's factors: U rows (kSweepUT: nc x fs), or L11 (the
  // first nc columns of the U rows, nc x nc) and L21 (uc x nc).
  template <SweepMode M>
  __device__ __forceinline__ void fetch_factors(T* buf, const int* w) const {
    const int shape = w[kSwShape], fs = shape & 0xffff, nc = shape >> 16;
    if constexpr (M == kSweepUT) {
      fetch(buf, a.U, (size_t)w[kSwU], nc * fs);
    } else {
      if (nc > 1)
        for (int k = 0; k < nc; ++k) fetch(buf + k * nc * S, a.U, (size_t)w[kSwU] + (size_t)k * fs, nc);
      fetch(buf + nc * nc * S, a.L, (size_t)w[kSwL], (fs - nc) * nc);
    }
  }

  // Solution rows of one front going down (k_sweep_down).  PW partial sums
  // per pivot, row j in sum (j - nc) % PW.
  template <int NC>
  __device__ __forceinline__ void solve_down(const int* w, int fs, const T* F, const T* y, T* x, T* part,
                                             const uint16_t* row, int PW) const {
    const int uc = fs - NC, lp = w[kSwLocal];
    const size_t first = (size_t)w[kSwFirst];
    for (int i = worker; i < NC * PW; i += Team::NW) {
      const int p = i / NC, k = i - p * NC;
      P r = pack_zero<T, V>();
#pragma unroll 4
      for (int j = p; j < uc; j += PW) {
        const P u = ld(F, NC * NC + j * NC + k), xv = ld(x, row[j]);
#pragma unroll
        for (int v = 0; v < V; ++v) r.x[v] += u.x[v] * xv.x[v];
      }
      st(part, i, r);
    }
    Team::sync();
    P s[NC];
#pragma unroll
    for (int k = NC - 1; k >= 0; --k) {
      s[k] = ld(y, k);
#pragma unroll
      for (int m = k + 1; m < NC; ++m) {
        const P u = ld(F, m * NC + k);
#pragma unroll
        for (int v = 0; v < V; ++v) s[k].x[v] -= u.x[v] * s[m].x[v];
      }
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < PW) {
          const P c = ld(part, p * NC + k);
#pragma unroll
          for (int v = 0; v < V; ++v) s[k].x[v] -= c.x[v];
        }
    }
#pragma unroll
    for (int k = 0; k < NC; ++k)
      if (k % Team::NW == worker) {
        st(x, lp + k, s[k]);
        out(a.X, first + k, s[k]);
      }
  }

  // Solution rows of one front going up, and its update vector (k_sweep_up).
  template <SweepMode M, int NC>
  __device__ __forceinline__ void solve_up(const int* w, int fs, const T* F, const T* y, const T* tr, T* arena) const {
    const int uc = fs - NC, tv = w[kSwTvArena];
    const size_t first = (size_t)w[kSwFirst];
    P s[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      s[k] = ld(y, k);
      const P c = ld(tr, k);
#pragma unroll
      for (int v = 0; v < V; ++v) s[k].x[v] -= c.x[v];
#pragma unroll
      for (int i = 0; i < k; ++i) {
        const P u = ld(F, M == kSweepUT ? i * fs + k : k * NC + i);
#pragma unroll
        for (int v = 0; v < V; ++v) s[k].x[v] -= u.x[v] * s[i].x[v];
      }
      if constexpr (M == kSweepUT) {
        const P d = ld(F, k * fs + k);
#pragma unroll
        for (int v = 0; v < V; ++v) s[k].x[v] = s[k].x[v] / d.x[v];
      }
      if (k % Team::NW == worker) out(a.W, first + k, s[k]);
    }
#pragma unroll 2
    for (int j = worker; j < uc; j += Team::NW) {
      P r = ld(tr, NC + j);
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const P u = ld(F, M == kSweepUT ? k * fs + NC + j : NC * NC + j * NC + k);
#pragma unroll
        for (int v = 0; v < V; ++v) r.x[v] += u.x[v] * s[k].x[v];
      }
      if (tv < 0) out(a.TV, (size_t)w[kSwTv] + j, r);
      else st(arena, tv + j, r);
    }
  }
};

__device__ __forceinline__ const uint16_t* sweep_lists(const int* w) {
  return reinterpret_cast<const uint16_t*>(w + w[kSwLists]);
}

// L^T z = w, one stage: a task's fronts from its root down.  The terms of the
// contribution rows are summed as the level kernels' warps sum them (their
// number follows from the front's level launch), then every worker solves the
// pivot block alike: the level kernels' order, so the solutions are the same
// bits.
// Shared memory of a team: x [local][S], a ring of factor buffers [max_f][S] and
// right-hand sides [8][S], partial sums [64][S].
template <typename T, int V, int LS, int TW>
__global__ void __launch_bounds__(TW == 1 ? 128 : TW * 32)
    k_sweep_down(SweepTaskArgs<T> a, const int* __restrict__ meta, const int* __restrict__ words, int groups,
                 int blocks_per_task, int prog_bytes, int max_local, int max_f, int groups32) {
  using Team = TaskTeam<T, V, LS, TW>;
  using P = Pack<T, V>;
  constexpr int S = Team::S, D = sweep_ring(TW);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_allow_next();
  const int t = blockIdx.x / blocks_per_task, bg = blockIdx.x - t * blocks_per_task;
  const int4 m = reinterpret_cast<const int4*>(meta)[t];
  int* prog = reinterpret_cast<int*>(smem_raw);
  for (int i = threadIdx.x; i < m.y / 4; i += blockDim.x) cp_async16(prog + 4 * i, words + m.x + 4 * i);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int team = TW == 1 ? (int)(threadIdx.x >> 5) : 0;
  const int grp = TW == 1 ? bg * (int)(blockDim.x >> 5) + team : bg;
  if (grp >= groups) return;
  const int tid = TW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const Sweeper<T, V, LS, TW> sw{a, (size_t)grp * S, tid, tid / LS, (tid % LS) * V};
  T* x = reinterpret_cast<T*>(smem_raw + prog_bytes) + (size_t)team * (max_local + D * (max_f + 8) + 64) * S;
  T* fb = x + (size_t)max_local * S;
  T* yb = fb + (size_t)D * max_f * S;
  T* part = yb + D * 8 * S;
  chain_wait_previous();  // factors, right-hand side, and the rows of earlier stages
  const int nf = m.z, nx = m.w;
  // external rows: the root's contribution rows, last in the local numbering
  const int root = prog[nf - 1];
  const int ext0 = prog[root + kSwLocal] + (prog[root + kSwShape] >> 16);
  {
    using R = Rows<T, S>;
    for (int i = tid; i < nx * R::kPieces; i += Team::NT) {
      const int j = i / R::kPieces, piece = (i % R::kPieces) * R::kPiece;
      R::fetch(reinterpret_cast<unsigned char*>(x + (size_t)(ext0 + j) * S) + piece,
               reinterpret_cast<const unsigned char*>(a.X + (size_t)prog[nf + j] * a.Bp + sw.col0) + piece);
    }
  }
  auto prefetch = [&](int f) {
    const int* w = prog + prog[f];
    sw.template fetch_factors<kSweepLT>(fb + (size_t)(f % D) * max_f * S, w);
    sw.fetch(yb + (size_t)(f % D) * 8 * S, a.W, (size_t)w[kSwFirst], w[kSwShape] >> 16);
    cp_async_commit();
  };
  for (int i = 1; i < D; ++i) {
    if (nf - i >= 0) prefetch(nf - i);
    else cp_async_commit();
  }
  for (int f = nf - 1; f >= 0; --f) {
    cp_async_wait<D - 2>();
    Team::sync();
    if (f >= D - 1) prefetch(f - (D - 1));
    else cp_async_commit();
    const int* w = prog + prog[f];
    const int shape = w[kSwShape], fs = shape & 0xffff, nc = shape >> 16;
    const T* F = fb + (size_t)(f % D) * max_f * S;
    const T* y = yb + (size_t)(f % D) * 8 * S;
    const uint16_t* row = sweep_lists(w);
    const int PW = sweep_warps((long)w[kSwLevel] * groups32);
    auto solve = [&](auto n) { sw.template solve_down<decltype(n)::value>(w, fs, F, y, x, part, row, PW); };
    switch (nc) {
      case 1: solve(std::integral_constant<int, 1>{}); break;
      case 2: solve(std::integral_constant<int, 2>{}); break;
      case 3: solve(std::integral_constant<int, 3>{}); break;
      case 4: solve(std::integral_constant<int, 4>{}); break;
      case 5: solve(std::integral_constant<int, 5>{}); break;
      case 6: solve(std::integral_constant<int, 6>{}); break;
      case 7: solve(std::integral_constant<int, 7>{}); break;
      default: solve(std::integral_constant<int, 8>{}); break;
    }
  }
}

// L y = b (M = kSweepL) or U^T w = g (kSweepUT), one stage: a task's fronts
// children first, in place in a.W (right-hand side in, solution out).  A
// front gathers its children's update vectors, solves its pivot block and
// emits its own vector: to the arena, or to a.TV at the task's root.
// Shared memory of a team: vectors [arena][S], gathered rows [max_rows][S],
// a ring of factor buffers [max_f][S] and right-hand sides [8][S].
template <SweepMode M, typename T, int V, int LS, int TW>
__global__ void __launch_bounds__(TW == 1 ? 128 : TW * 32)
    k_sweep_up(SweepTaskArgs<T> a, const int* __restrict__ meta, const int* __restrict__ words, int groups,
               int blocks_per_task, int prog_bytes, int max_arena, int max_rows, int max_f) {
  using Team = TaskTeam<T, V, LS, TW>;
  using P = Pack<T, V>;
  constexpr int S = Team::S, D = sweep_ring(TW);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_allow_next();
  const int t = blockIdx.x / blocks_per_task, bg = blockIdx.x - t * blocks_per_task;
  const int4 m = reinterpret_cast<const int4*>(meta)[t];
  int* prog = reinterpret_cast<int*>(smem_raw);
  for (int i = threadIdx.x; i < m.y / 4; i += blockDim.x) cp_async16(prog + 4 * i, words + m.x + 4 * i);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int team = TW == 1 ? (int)(threadIdx.x >> 5) : 0;
  const int grp = TW == 1 ? bg * (int)(blockDim.x >> 5) + team : bg;
  if (grp >= groups) return;
  const int tid = TW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const Sweeper<T, V, LS, TW> sw{a, (size_t)grp * S, tid, tid / LS, (tid % LS) * V};
  T* arena = reinterpret_cast<T*>(smem_raw + prog_bytes) + (size_t)team * (max_arena + max_rows + D * (max_f + 8)) * S;
  T* tr = arena + (size_t)max_arena * S;
  T* fb = tr + (size_t)max_rows * S;
  T* yb = fb + (size_t)D * max_f * S;
  chain_wait_previous();  // factors, right-hand side, and the vectors of earlier stages
  const int nf = m.z;
  auto prefetch = [&](int f) {
    const int* w = prog + prog[f];
    const int* ext = w + kSweepRecordWords + w[kSwPass];
    sw.template fetch_factors<M>(fb + (size_t)(f % D) * max_f * S, w);
    sw.fetch(yb + (size_t)(f % D) * 8 * S, a.W, (size_t)w[kSwFirst], w[kSwShape] >> 16);
    for (int c = 0; c < w[kSwExt]; ++c)
      sw.fetch(arena + (size_t)ext[3 * c + 2] * S, a.TV, (size_t)ext[3 * c], ext[3 * c + 1]);
    cp_async_commit();
  };
  for (int i = 0; i < D - 1; ++i) {
    if (i < nf) prefetch(i);
    else cp_async_commit();
  }
  for (int f = 0; f < nf; ++f) {
    cp_async_wait<D - 2>();
    Team::sync();
    const int* w = prog + prog[f];
    const int shape = w[kSwShape], fs = shape & 0xffff, nc = shape >> 16, uc = fs - nc, npass = w[kSwPass];
    const int* count = w + kSweepRecordWords;
    const uint16_t* row = sweep_lists(w) + uc;
    const uint16_t* src = row + fs;
    for (int i = sw.worker; i < fs; i += Team::NW) {
      P s = pack_zero<T, V>();
      const uint16_t* q = src;
      for (int p = 0; p < npass; ++p) {
        const int n = count[p];
        if (i >= n) break;
        const P c = sw.ld(arena, q[i]);
#pragma unroll
        for (int v = 0; v < V; ++v) s.x[v] += c.x[v];
        q += n;
      }
      sw.st(tr, row[i], s);
    }
    Team::sync();
    if (f + D - 1 < nf) prefetch(f + D - 1);
    else cp_async_commit();
    const T* F = fb + (size_t)(f % D) * max_f * S;
    const T* y = yb + (size_t)(f % D) * 8 * S;
    auto solve = [&](auto n) { sw.template solve_up<M, decltype(n)::value>(w, fs, F, y, tr, arena); };
    switch (nc) {
      case 1: solve(std::integral_constant<int, 1>{}); break;
      case 2: solve(std::integral_constant<int, 2>{}); break;
      case 3: solve(std::integral_constant<int, 3>{}); break;
      case 4: solve(std::integral_constant<int, 4>{}); break;
      case 5: solve(std::integral_constant<int, 5>{}); break;
      case 6: solve(std::integral_constant<int, 6>{}); break;
      case 7: solve(std::integral_constant<int, 7>{}); break;
      default: solve(std::integral_constant<int, 8>{}); break;
    }
  }
}

template <SweepMode M, typename T, int V, int LS, int TW>
void launch_sweep_tasks(const SweepTaskStage& st, const SweepTaskArgs<T>& a, int groups32, const int* meta,
                        const int* words, int lanes, cudaStream_t s) {
  using Team = TaskTeam<T, V, LS, TW>;
  const int groups = (lanes + Team::S - 1) / Team::S;
  const size_t prog = (size_t)(st.max_words + 3) / 4 * 16;
  constexpr bool kDown = M == kSweepLT;
  const int max_f = (M == kSweepL || M == kSweepLT) ? 64 + st.max_l : st.max_u;
  const size_t elems = (kDown ? (size_t)st.max_local + 64 : (size_t)st.max_arena + st.max_rows) +
                       (size_t)sweep_ring(TW) * (max_f + 8);
  const size_t team = elems * Team::S * sizeof(T);
  int teams = 1;
  if (TW == 1) teams = teams_per_block(groups, prog, team);
  const int blocks_per_task = (groups + teams - 1) / teams;
  const size_t smem = prog + teams * team;
  if (smem > kSmemLimit) throw std::runtime_error("sweep tasks: a task exceeds shared memory");
  const dim3 grid((unsigned)(st.count * blocks_per_task)), block(TW == 1 ? teams * 32 : TW * 32);
  meta += 4 * (size_t)st.begin;
  if constexpr (kDown) {
    auto kern = k_sweep_down<T, V, LS, TW>;
    allow_full_smem(reinterpret_cast<const void*>(kern));
    launch_chained(kern, grid, block, smem, s, "sweep tasks", a, meta, words, groups, blocks_per_task, (int)prog,
                   st.max_local, max_f, groups32);
  } else {
    auto kern = k_sweep_up<M, T, V, LS, TW>;
    allow_full_smem(reinterpret_cast<const void*>(kern));
    launch_chained(kern, grid, block, smem, s, "sweep tasks", a, meta, words, groups, blocks_per_task, (int)prog,
                   st.max_arena, st.max_rows, max_f);
  }
}

}  // namespace

template <typename T>
void launch_sweep_stage(int mode, const SweepTaskStage& st, const SweepTaskArgs<T>& a, int groups, const int* meta,
                        const int* words, int lanes, cudaStream_t s) {
  auto run = [&](auto m) {
    constexpr SweepMode M = decltype(m)::value;
    if (lanes == 1) {  // a single system: every thread a worker
      if (st.warps > 1) launch_sweep_tasks<M, T, 1, 1, 2>(st, a, groups, meta, words, lanes, s);
      else launch_sweep_tasks<M, T, 1, 1, 1>(st, a, groups, meta, words, lanes, s);
      return;
    }
    // the shapes sweep_task_specs uses (block teams take 4 scenarios in FP64:
    // the specs' limits fill shared memory with 4 x 8 and 8 x 4 bytes alike)
    if (st.warps == 2 && st.lanes == 8 && st.pack == 1)
      launch_sweep_tasks<M, T, 1, sizeof(T) == 8 ? 4 : 8, 2>(st, a, groups, meta, words, lanes, s);
    else if (st.warps == 1 && st.lanes == 16 && st.pack == 1)
      launch_sweep_tasks<M, T, 1, 16, 1>(st, a, groups, meta, words, lanes, s);
    else if (st.warps == 1 && st.lanes == 8 && st.pack == 1)
      launch_sweep_tasks<M, T, 1, 8, 1>(st, a, groups, meta, words, lanes, s);
    else
      throw std::runtime_error("sweep tasks: no kernel for teams of " + std::to_string(st.warps) + " warps, " +
                               std::to_string(st.lanes) + " lanes, " + std::to_string(st.pack) + " scenarios a lane");
  };
  switch (mode) {
    case kSweepL: run(std::integral_constant<SweepMode, kSweepL>{}); break;
    case kSweepUT: run(std::integral_constant<SweepMode, kSweepUT>{}); break;
    default: run(std::integral_constant<SweepMode, kSweepLT>{}); break;
  }
}

}  // namespace cupf_b200
