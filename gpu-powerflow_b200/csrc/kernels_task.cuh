// kernels_task.cuh -- factorization of whole subtrees of fronts (task_plan.hpp).
//
// The level kernels (kernels_lu.cuh) launch once per level of the front tree
// and give each front of 32 scenarios a block: a front of 3 to 8 rows, which
// most are, then costs a chain of memory round trips for a few hundred
// operations, and every contribution block travels through global memory.
// Here a team of threads factors a whole subtree for S scenarios.  Its
// program (the list of its fronts with their assembly lists) is fetched once;
// the next front's Jacobian entries arrive by cp.async while the current one
// is eliminated; contribution blocks pass from child to parent in shared
// memory.  Lanes: LS lanes x V scenarios cover the S = LS * V scenarios, and
// the 32 / LS groups of a warp ("workers") share out a front's elements, so
// small batches still use every lane of a warp.
//
// What bounds it: instruction issue and latency, not memory (2,000 buses
// x 1,024 FP32, first stage to last: 11, 12, 7, 5 and 8 resident warps on an SM,
// which the arenas' shared memory and the registers limit; 47, 47, 28, 29 and
// 32 % of issue slots used; DRAM at 27, 14, 6, 3 and 2 %), hence several
// scenarios per lane, unrolled small fronts, and joined subtrees that fill the
// pipeline once per block instead of once per subtree (first stage 101 -> 58 us).
// Measured per factorization, level launches -> tasks: 2,000 buses x 1,024
// FP32 521 -> 293 us and FP64 760 -> 488 us, 10,000 x 64 FP32 540 -> 209 us,
// 2,000 x 1 140 -> 105 us.
//
// Every element sees the operations of the level kernels in the same order
// (sources: Jacobian entry, then children ascending; pivots ascending;
// multiplier = value times the pivot's reciprocal), so the factors are the
// same bits.
#pragma once

#include <algorithm>
#include <cstdint>

#include "kernel_util.cuh"
#include "task_plan.hpp"

namespace cupf_b200 {
namespace {

template <typename T, int V>
struct alignas(sizeof(T) * V) Pack {
  T x[V];
};

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> pack_zero() {
  Pack<T, V> r;
#pragma unroll
  for (int v = 0; v < V; ++v) r.x[v] = T(0);
  return r;
}

// Stages one row of S scenarios in 16-byte pieces (S = 1: one element).
template <typename T, int S>
struct Rows {
  static constexpr int kBytes = S * (int)sizeof(T);
  static constexpr int kPiece = kBytes >= 16 ? 16 : kBytes;
  static constexpr int kPieces = kBytes / kPiece;
  static __device__ __forceinline__ void fetch(unsigned char* smem, const void* gmem) {
    if constexpr (kPiece == 16) cp_async16(smem, gmem);
    else if constexpr (kPiece == 8) cp_async8(smem, gmem);
    else cp_async4(smem, gmem);
  }
  static __device__ __forceinline__ void zero(unsigned char* smem) {
    if constexpr (kPiece == 16) *reinterpret_cast<float4*>(smem) = make_float4(0.f, 0.f, 0.f, 0.f);
    else if constexpr (kPiece == 8) *reinterpret_cast<float2*>(smem) = make_float2(0.f, 0.f);
    else *reinterpret_cast<float*>(smem) = 0.f;
  }
};

// TW: warps of a team.  TW = 1: a block holds several teams (one task, one
// scenario group per warp), which share nothing but the program; TW > 1: the
// block is the team.
template <typename T, int V, int LS, int TW>
struct TaskTeam {
  static constexpr int S = LS * V;          // scenarios
  static constexpr int NW = TW * 32 / LS;   // workers
  static constexpr int NT = TW * 32;        // threads
  // workers over a front's rows and columns: pivot rows x columns, and
  // non-pivot rows x columns
  static constexpr int WJ = NW <= 4 ? NW : NW <= 32 ? 8 : 16;
  static constexpr int WI = NW / WJ;
  static constexpr int NR = NW <= 8 ? NW : NW <= 16 ? 8 : 16;
  static constexpr int NC = NW / NR;
  static __device__ __forceinline__ void sync() {
    if constexpr (TW == 1) __syncwarp();
    else __syncthreads();
  }
};

template <typename T, int V, int LS, int TW>
struct FrontTask {
  using Team = TaskTeam<T, V, LS, TW>;
  using P = Pack<T, V>;
  using R = Rows<T, Team::S>;
  static constexpr int S = Team::S;

  const FactorArgs<T, T>& a;
  T* arena;  // this team's, [element][S]
  T* inv;    // [8][S] pivot reciprocals
  size_t col0;
  int tid, worker, s0;
  unsigned shifted = 0;  // bit v: a pivot of this lane's scenario v was replaced

  __device__ __forceinline__ P ld(const T* base, int e) const {
    return *reinterpret_cast<const P*>(base + e * S + s0);
  }
  __device__ __forceinline__ void st(T* base, int e, const P& v) const { *reinterpret_cast<P*>(base + e * S + s0) = v; }
  // a value into this team's columns of a [element][Bp] array
  __device__ __forceinline__ void out(T* g, size_t e, const P& v) const {
    *reinterpret_cast<P*>(g + e * a.Bp + col0 + s0) = v;
  }

  struct Lists {
    const int *count, *ext, *jsrc;
    const unsigned* term;
    const uint16_t *jdst, *zdst;
    int nj, nz, npass, next;
  };
  static __device__ __forceinline__ Lists lists(const int* w) {
    Lists l;
    const unsigned j = (unsigned)w[kTwJ];
    l.nj = j & 0xffff;
    l.nz = j >> 16;
    l.npass = w[kTwPass];
    l.next = w[kTwExt];
    l.count = w + kTaskRecordWords;
    l.ext = l.count + l.npass;
    l.jsrc = l.ext + 3 * l.next;
    l.term = reinterpret_cast<const unsigned*>(l.jsrc + l.nj);
    l.jdst = reinterpret_cast<const uint16_t*>(w + w[kTwHalf]);
    l.zdst = l.jdst + l.nj;
    return l;
  }

  // Fills front w's buffer: its Jacobian and right-hand-side entries and the
  // contribution blocks of children outside the task (asynchronous), zeros
  // elsewhere.
  __device__ __forceinline__ void fetch(const int* w) {
    const Lists l = lists(w);
    const int shape = w[kTwShape], fs = shape & 0xff, nc = (shape >> 8) & 0xff, rs = task_front_stride(fs);
    unsigned char* F = reinterpret_cast<unsigned char*>(arena + (size_t)w[kTwFront] * S);
    constexpr int PP = R::kPieces;
    const size_t cb = col0 * sizeof(T);
    const unsigned char* J = reinterpret_cast<const unsigned char*>(a.J) + cb;
    const size_t row = (size_t)a.Bp * sizeof(T);
    for (int i = tid; i < l.nj * PP; i += Team::NT) {
      const int e = i / PP, piece = (i % PP) * R::kPiece;
      R::fetch(F + (int)l.jdst[e] * R::kBytes + piece, J + (size_t)l.jsrc[e] * row + piece);
    }
    const unsigned char* Fp = reinterpret_cast<const unsigned char*>(a.Fp) + cb;
    for (int i = tid; i < nc * PP; i += Team::NT) {
      const int k = i / PP, piece = (i % PP) * R::kPiece;
      R::fetch(F + (k * rs + fs) * R::kBytes + piece, Fp + (size_t)(w[kTwFirst] + k) * row + piece);
    }
    const unsigned char* C = reinterpret_cast<const unsigned char*>(a.CB) + cb;
    for (int c = 0; c < l.next; ++c) {
      const int co = l.ext[3 * c], n = l.ext[3 * c + 1];
      unsigned char* X = reinterpret_cast<unsigned char*>(arena + (size_t)l.ext[3 * c + 2] * S);
      for (int i = tid; i < n * PP; i += Team::NT) {
        const int e = i / PP, piece = (i % PP) * R::kPiece;
        R::fetch(X + e * R::kBytes + piece, C + (size_t)(co + e) * row + piece);
      }
    }
    cp_async_commit();
    for (int i = tid; i < l.nz * PP; i += Team::NT)
      R::zero(F + (int)l.zdst[i / PP] * R::kBytes + (i % PP) * R::kPiece);
  }

  // The children's terms, pass by pass: a destination has the same place in
  // every pass, so one worker adds its terms, in child order.
  __device__ __forceinline__ void assemble(const int* w) {
    const Lists l = lists(w);
    T* F = arena + (size_t)w[kTwFront] * S;
    const unsigned* q = l.term;
    for (int p = 0; p < l.npass; ++p) {
      const int n = l.count[p];
#pragma unroll(TW == 1 ? 4 : 8)
      for (int x = worker; x < n; x += Team::NW) {
        const unsigned ds = q[x];
        P v = ld(F, ds & 0xffff);
        const P t = ld(arena, ds >> 16);
#pragma unroll
        for (int k = 0; k < V; ++k) v.x[k] += t.x[k];
        st(F, ds & 0xffff, v);
      }
      q += n;
    }
  }

  // Guards the pivot at element e of the front and keeps its reciprocal in
  // inv[k]: worker v takes scenario v of a lane's V.
  __device__ __forceinline__ T guard(T p, int v) {
    bool sh = false;
    p = guarded_pivot(p, a.static_pivot != 0, a.eps, sh);
    if (sh) shifted |= 1u << v;
    return p;
  }

  // Elimination of a front of up to 8 rows and 4 pivots by a warp (most
  // fronts), a lane per scenario: the pivot rows in registers, all 9 columns
  // at fixed offsets (columns past fs hold nothing that is stored), the other
  // rows one after the other over the 32 / S lanes of a scenario.
  template <int NC_>
  __device__ __forceinline__ void eliminate_lanes(const int* w, int fs, T* F) {
    constexpr int RS = kSmallFront + 1, NL = 32 / S;
    const int sc = tid % S, wl = tid / S;
    T* f = F + sc;
    const size_t b = col0 + sc, Bp = a.Bp;
    const int uc = fs - NC_;
    T u[NC_][RS], iv[NC_];
#pragma unroll
    for (int k = 0; k < NC_; ++k)
#pragma unroll
      for (int j = 0; j < RS; ++j) u[k][j] = f[(k * RS + j) * S];
    bool sh = false;
#pragma unroll
    for (int k = 0; k < NC_; ++k) {
#pragma unroll
      for (int m = 0; m < k; ++m) {
        u[k][m] *= iv[m];
#pragma unroll
        for (int j = m + 1; j < RS; ++j) u[k][j] -= u[k][m] * u[m][j];
      }
      u[k][k] = guarded_pivot(u[k][k], a.static_pivot != 0, a.eps, sh);
      iv[k] = T(1) / u[k][k];
    }
    if (sh) a.sing[b] = 1;
    const bool leaves = (w[kTwShape] >> 16) != 0;
    T* C = leaves ? a.CB + (size_t)w[kTwCb] * Bp + b : arena + (size_t)w[kTwCbArena] * S + sc;
    const size_t cs = leaves ? Bp : (size_t)S;
    for (int ii = wl; ii < uc; ii += NL) {
      T r[RS];
#pragma unroll
      for (int j = 0; j < RS; ++j) r[j] = f[((NC_ + ii) * RS + j) * S];
#pragma unroll
      for (int m = 0; m < NC_; ++m) {
        r[m] *= iv[m];
#pragma unroll
        for (int j = m + 1; j < RS; ++j) r[j] -= r[m] * u[m][j];
      }
      T* Ci = C + (size_t)(ii * (uc + 1)) * cs;
#pragma unroll
      for (int j = NC_; j < RS; ++j)
        if (j <= fs) Ci[(j - NC_) * cs] = r[j];
      if (a.store_l) {
#pragma unroll
        for (int m = 0; m < NC_; ++m) a.L[((size_t)w[kTwL] + (size_t)ii * NC_ + m) * Bp + b] = r[m];
      }
    }
    // U rows and y (every lane of a scenario holds them; rows over the lanes)
    T* Ub = a.U + (size_t)w[kTwU] * Bp + b;
    T* Yb = a.Y + (size_t)w[kTwFirst] * Bp + b;
#pragma unroll
    for (int k = 0; k < NC_; ++k)
      if (k % NL == wl) {
#pragma unroll
        for (int j = 0; j < RS; ++j) {
          if (j < fs) Ub[((size_t)k * fs + j) * Bp] = u[k][j];
          if (j == fs) Yb[(size_t)k * Bp] = u[k][j];
        }
      }
  }

  // Elimination of a larger front with one or two pivots by a warp:
  // the pivot block by one worker per scenario, then no barrier is needed --
  // a worker updates the second pivot row's entries as it meets them.
  template <int NC_>
  __device__ __forceinline__ void eliminate_small(const int* w, int fs, int rs, T* F) {
    if (worker < V) {
      T* f = F + s0 + worker;
      T* iv = inv + s0 + worker;
      const T p0 = guard(f[0], worker);
      const T i0 = T(1) / p0;
      f[0] = p0;
      iv[0] = i0;
      if constexpr (NC_ == 2) {
        const T l10 = f[rs * S] * i0;
        const T p1 = guard(f[(rs + 1) * S] - l10 * f[S], worker);
        f[rs * S] = l10;
        f[(rs + 1) * S] = p1;
        iv[S] = T(1) / p1;
      }
    }
    __syncwarp();
    const P i0 = ld(inv, 0);
    P i1, l10, u01;
    if constexpr (NC_ == 2) {
      i1 = ld(inv, 1);
      l10 = ld(F, rs);
      u01 = ld(F, 1);
    }
    const int uc = fs - NC_;
    const bool leaves = (w[kTwShape] >> 16) != 0;
    T* C = leaves ? a.CB + (size_t)w[kTwCb] * a.Bp + col0 + s0 : arena + (size_t)w[kTwCbArena] * S + s0;
    const size_t cs = leaves ? (size_t)a.Bp : (size_t)S;
    for (int ii = worker; ii < uc; ii += Team::NW) {
      const T* Fi = F + (NC_ + ii) * rs * S;
      P l0 = ld(Fi, 0), l1;
#pragma unroll
      for (int k = 0; k < V; ++k) l0.x[k] *= i0.x[k];
      if constexpr (NC_ == 2) {
        l1 = ld(Fi, 1);
#pragma unroll
        for (int k = 0; k < V; ++k) l1.x[k] = (l1.x[k] - l0.x[k] * u01.x[k]) * i1.x[k];
      }
      if (a.store_l) {
        out(a.L, (size_t)w[kTwL] + (size_t)ii * NC_, l0);
        if constexpr (NC_ == 2) out(a.L, (size_t)w[kTwL] + (size_t)ii * NC_ + 1, l1);
      }
      T* Ci = C + (size_t)(ii * (uc + 1)) * cs;
#pragma unroll 4
      for (int j = NC_; j <= fs; ++j, Ci += cs) {
        P r = ld(Fi, j);
        const P u0 = ld(F, j);
#pragma unroll
        for (int k = 0; k < V; ++k) r.x[k] -= l0.x[k] * u0.x[k];
        if constexpr (NC_ == 2) {
          P u1 = ld(F, rs + j);
#pragma unroll
          for (int k = 0; k < V; ++k) u1.x[k] -= l10.x[k] * u0.x[k];
#pragma unroll
          for (int k = 0; k < V; ++k) r.x[k] -= l1.x[k] * u1.x[k];
        }
        *reinterpret_cast<P*>(Ci) = r;
      }
    }
    // U rows and y: the pivot block as stored, then the rows' other columns
    const size_t uo = (size_t)w[kTwU], first = (size_t)w[kTwFirst];
    for (int j = worker; j <= fs; j += Team::NW) {
      const P u0 = ld(F, j);
      if (j < fs) out(a.U, uo + j, u0);
      else out(a.Y, first, u0);
      if constexpr (NC_ == 2) {
        P u1 = ld(F, rs + j);
        if (j >= 2) {
#pragma unroll
          for (int k = 0; k < V; ++k) u1.x[k] -= l10.x[k] * u0.x[k];
        }
        if (j < fs) out(a.U, uo + fs + j, u1);
        else out(a.Y, first + 1, u1);
      }
    }
  }

  // The pivot block [nc][nc], right-looking, by a one-warp team; leaves
  // the multipliers, the guarded pivots and U there, reciprocals in inv.
  __device__ __forceinline__ void pivot_block(int nc, int rs, T* F) {
    constexpr int W1 = 32 / LS;  // workers of a warp
    for (int k = 0; k < nc; ++k) {
      if (k > 0) __syncwarp();
      if constexpr (V == 1) {
        const T p = guard(F[(k * rs + k) * S + s0], 0), iv = T(1) / p;
        __syncwarp();  // every lane has read the pivot
        if (worker == 0) {
          F[(k * rs + k) * S + s0] = p;
          inv[k * S + s0] = iv;
        }
      } else if (worker < V) {
        T* f = F + (k * rs + k) * S + s0 + worker;
        const T p = guard(*f, worker);
        *f = p;
        inv[k * S + s0 + worker] = T(1) / p;
      }
      __syncwarp();
      const P iv = ld(inv, k);
      const int n = nc - 1 - k;
      for (int i = k + 1 + (worker / 8); i < nc; i += (W1 + 7) / 8) {
        P l = ld(F, i * rs + k);
#pragma unroll
        for (int v = 0; v < V; ++v) l.x[v] *= iv.x[v];
        for (int j = worker % 8; j < n; j += (W1 < 8 ? W1 : 8)) {
          P r = ld(F, i * rs + k + 1 + j);
          const P u = ld(F, k * rs + k + 1 + j);
#pragma unroll
          for (int v = 0; v < V; ++v) r.x[v] -= l.x[v] * u.x[v];
          st(F, i * rs + k + 1 + j, r);
        }
      }
      __syncwarp();  // every lane has read the column's unscaled entries
      for (int i = k + 1 + worker; i < nc; i += W1) {
        P l = ld(F, i * rs + k);
#pragma unroll
        for (int v = 0; v < V; ++v) l.x[v] *= iv.x[v];
        st(F, i * rs + k, l);
      }
    }
  }

  // Row multipliers (L21) and the pivot rows' other columns (U12 | y) from
  // the finished pivot block, one row or column per worker; nc <= NCB.
  template <int NCB>
  __device__ __forceinline__ void panels(const int* w, int fs, int nc, int rs, T* F) {
    constexpr int W1 = 32 / LS;
    const int uc = fs - nc, rows = (uc + W1 - 1) / W1 * W1;  // (a warp takes rows or columns)
    for (int t = worker; t < rows + uc + 1; t += Team::NW) {
      P x[NCB];
      if (t < rows) {
        if (t >= uc) continue;
        T* Fi = F + (nc + t) * rs * S;
#pragma unroll
        for (int m = 0; m < NCB; ++m)
          if (m < nc) {
            P r = ld(Fi, m);
#pragma unroll
            for (int q = 0; q < NCB; ++q)
              if (q < m) {
                const P u = ld(F, q * rs + m);
#pragma unroll
                for (int v = 0; v < V; ++v) r.x[v] -= x[q].x[v] * u.x[v];
              }
            const P iv = ld(inv, m);
#pragma unroll
            for (int v = 0; v < V; ++v) x[m].x[v] = r.x[v] * iv.x[v];
            st(Fi, m, x[m]);
            if (a.store_l) out(a.L, (size_t)w[kTwL] + (size_t)t * nc + m, x[m]);
          }
      } else {
        T* Fj = F + (nc + t - rows) * S;
#pragma unroll
        for (int m = 0; m < NCB; ++m)
          if (m < nc) {
            x[m] = ld(Fj, m * rs);
#pragma unroll
            for (int q = 0; q < NCB; ++q)
              if (q < m) {
                const P l = ld(F, m * rs + q);
#pragma unroll
                for (int v = 0; v < V; ++v) x[m].x[v] -= l.x[v] * x[q].x[v];
              }
            if (m > 0) st(Fj, m * rs, x[m]);
          }
      }
    }
  }

  // Contribution block = trailing block - L21 U12, a worker per row and
  // every NC-th column; nc <= NCB.
  template <int NCB>
  __device__ __forceinline__ void trailing(const int* w, int fs, int nc, int rs, const T* F) {
    const int uc = fs - nc;
    const bool leaves = (w[kTwShape] >> 16) != 0;
    T* C = leaves ? a.CB + (size_t)w[kTwCb] * a.Bp + col0 + s0 : arena + (size_t)w[kTwCbArena] * S + s0;
    const size_t cs = leaves ? (size_t)a.Bp : (size_t)S;
    const int wr = worker / Team::NC, wc = worker % Team::NC;
    for (int ii = wr; ii < uc; ii += Team::NR) {
      const T* Fi = F + (nc + ii) * rs * S;
      P l[NCB];
#pragma unroll
      for (int m = 0; m < NCB; ++m)
        if (m < nc) l[m] = ld(Fi, m);
      T* Ci = C + (size_t)(ii * (uc + 1) + wc) * cs;
#pragma unroll 2
      for (int j = nc + wc; j <= fs; j += Team::NC, Ci += Team::NC * cs) {
        P r = ld(Fi, j);
#pragma unroll
        for (int m = 0; m < NCB; ++m)
          if (m < nc) {
            const P u = ld(F, m * rs + j);
#pragma unroll
            for (int v = 0; v < V; ++v) r.x[v] -= l[m].x[v] * u.x[v];
          }
        *reinterpret_cast<P*>(Ci) = r;
      }
    }
  }

  // Elimination with the pivot block in registers (nc <= NCB): every worker
  // factors it for itself (no barrier until the panels are done), then takes
  // rows of L21 and columns of U12 as panels() does.  With a constant nc the
  // bounds fold away; the larger teams use one instance for all nc, because a
  // launch at the top of the tree runs a few fronts per SM and each further
  // instance would be fetched cold by its first front.
  template <int NCB>
  __device__ __forceinline__ void eliminate_regs(const int* w, int fs, int nc, int rs, T* F) {
    constexpr int W1 = 32 / LS;
    const size_t uo = (size_t)w[kTwU], first = (size_t)w[kTwFirst];
    {
      P b[NCB][NCB], iv[NCB];
#pragma unroll
      for (int i = 0; i < NCB; ++i)
#pragma unroll
        for (int j = 0; j < NCB; ++j) b[i][j] = i < nc && j < nc ? ld(F, i * rs + j) : pack_zero<T, V>();
#pragma unroll
      for (int k = 0; k < NCB; ++k) {
        if (k >= nc) break;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          b[k][k].x[v] = guard(b[k][k].x[v], v);
          iv[k].x[v] = T(1) / b[k][k].x[v];
        }
#pragma unroll
        for (int i = k + 1; i < NCB; ++i)
#pragma unroll
          for (int v = 0; v < V; ++v) {
            b[i][k].x[v] *= iv[k].x[v];
#pragma unroll
            for (int j = k + 1; j < NCB; ++j) b[i][j].x[v] -= b[i][k].x[v] * b[k][j].x[v];
          }
        if (k % Team::NW == worker) {
#pragma unroll
          for (int j = 0; j < NCB; ++j)
            if (j < nc) out(a.U, uo + (size_t)k * fs + j, b[k][j]);
        }
      }
      const int uc = fs - nc, rows = (uc + W1 - 1) / W1 * W1;  // (a warp takes rows or columns)
      for (int t = worker; t < rows + uc + 1; t += Team::NW) {
        P x[NCB];
        if (t < rows) {
          if (t >= uc) continue;
          T* Fi = F + (nc + t) * rs * S;
#pragma unroll
          for (int m = 0; m < NCB; ++m)
            if (m < nc) x[m] = ld(Fi, m);
#pragma unroll
          for (int m = 0; m < NCB; ++m) {
            if (m >= nc) break;
#pragma unroll
            for (int v = 0; v < V; ++v) {
#pragma unroll
              for (int q = 0; q < m; ++q) x[m].x[v] -= x[q].x[v] * b[q][m].x[v];
              x[m].x[v] *= iv[m].x[v];
            }
            st(Fi, m, x[m]);
            if (a.store_l) out(a.L, (size_t)w[kTwL] + (size_t)t * nc + m, x[m]);
          }
        } else {
          const int j = nc + t - rows;
          const bool rhs = j == fs;
          T* g = rhs ? a.Y + first * a.Bp : a.U + (uo + j) * a.Bp;
          const size_t gs = (rhs ? (size_t)1 : (size_t)fs) * a.Bp;
#pragma unroll
          for (int m = 0; m < NCB; ++m)
            if (m < nc) x[m] = ld(F, m * rs + j);
#pragma unroll
          for (int m = 0; m < NCB; ++m) {
            if (m >= nc) break;
#pragma unroll
            for (int q = 0; q < m; ++q)
#pragma unroll
              for (int v = 0; v < V; ++v) x[m].x[v] -= b[m][q].x[v] * x[q].x[v];
            if (m > 0) st(F, m * rs + j, x[m]);
            *reinterpret_cast<P*>(g + m * gs + col0 + s0) = x[m];
          }
        }
      }
    }
    Team::sync();
    trailing<NCB>(w, fs, nc, rs, F);
  }

  // The same through shared memory: five pivots and more in a one-warp team,
  // whose launches would lose resident teams to the registers.
  __device__ __forceinline__ void eliminate_shared(const int* w, int fs, int nc, int rs, T* F) {
    static_assert(TW == 1, "one-warp teams");
    pivot_block(nc, rs, F);
    Team::sync();
    panels<8>(w, fs, nc, rs, F);
    Team::sync();
    trailing<8>(w, fs, nc, rs, F);
    // U rows (multipliers | pivot | U) and y
    const size_t uo = (size_t)w[kTwU];
    const int wi = worker / Team::WJ, wj = worker % Team::WJ;
    for (int k = wi; k < nc; k += Team::WI) {
#pragma unroll 2
      for (int j = wj; j < fs; j += Team::WJ) out(a.U, uo + (size_t)k * fs + j, ld(F, k * rs + j));
    }
    for (int k = worker; k < nc; k += Team::NW) out(a.Y, (size_t)w[kTwFirst] + k, ld(F, k * rs + fs));
  }

  __device__ __forceinline__ void eliminate(const int* w) {
    const int shape = w[kTwShape], fs = shape & 0xff, nc = (shape >> 8) & 0xff, rs = task_front_stride(fs);
    T* F = arena + (size_t)w[kTwFront] * S;
    if constexpr (TW == 1) {
      switch (nc) {
        case 1: return fs <= kSmallFront ? eliminate_lanes<1>(w, fs, F) : eliminate_small<1>(w, fs, rs, F);
        case 2: return fs <= kSmallFront ? eliminate_lanes<2>(w, fs, F) : eliminate_small<2>(w, fs, rs, F);
        case 3: return eliminate_regs<3>(w, fs, 3, rs, F);
        case 4: return eliminate_regs<4>(w, fs, 4, rs, F);
        default: return eliminate_shared(w, fs, nc, rs, F);
      }
    } else if constexpr (TW == 2) {
      switch (nc) {
        case 1: return eliminate_regs<1>(w, fs, 1, rs, F);
        case 2: return eliminate_regs<2>(w, fs, 2, rs, F);
        case 3: return eliminate_regs<3>(w, fs, 3, rs, F);
        case 4: return eliminate_regs<4>(w, fs, 4, rs, F);
        case 8: return eliminate_regs<8>(w, fs, 8, rs, F);
        default: return eliminate_regs<8>(w, fs, nc, rs, F);
      }
    } else {
      eliminate_regs<8>(w, fs, nc, rs, F);
    }
  }
};

// Blocks per SM the register allocation allows for: bottom launches keep as
// many one-warp teams resident as their arenas leave room for.
constexpr int team_blocks(int elem, int v, int tw) {
  return tw > 1 ? 1 : elem == 8 ? (v == 1 ? 4 : v == 2 ? 3 : 2) : v == 1 ? 8 : v == 2 ? 6 : 4;
}

// One launch factors the tasks of a stage: block (task, scenario groups).
// TW = 1: warp w of a block takes group blockgroup * warps + w.
template <typename T, int V, int LS, int TW>
__global__ void __launch_bounds__(TW == 1 ? 128 : TW * 32, team_blocks(sizeof(T), V, TW))
    k_factor_tasks(FactorArgs<T, T> a, const int* __restrict__ meta, const int* __restrict__ words, int groups,
                   int blocks_per_task, int prog_bytes, int arena_elems) {
  using Task = FrontTask<T, V, LS, TW>;
  using Team = typename Task::Team;
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
  if (grp >= groups) return;  // (whole warps; nothing below spans the teams of a block)
  const int tid = TW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  T* mine = reinterpret_cast<T*>(smem_raw + prog_bytes) + (size_t)team * (arena_elems + 8) * Team::S;
  Task task{a, mine + 8 * Team::S, mine, (size_t)grp * Team::S, tid, tid / LS, (tid % LS) * V};
  chain_wait_previous();  // J, Fp and the blocks of earlier stages
  const int* w = prog;
  task.fetch(w);
  for (int f = 0; f < m.z; ++f) {
    cp_async_wait<0>();
    Team::sync();
    task.assemble(w);
    Team::sync();
    const int* next = w + w[kTwNext];
    if (f + 1 < m.z) task.fetch(next);
    task.eliminate(w);
    w = next;
  }
  if (task.shifted) {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (task.shifted >> v & 1) a.sing[task.col0 + task.s0 + v] = 1;
  }
}

}  // namespace

// Teams of one warp in a block: as many (up to 4, to share a program) as keep
// the most teams resident in an SM's shared memory.
inline int teams_per_block(int groups, size_t prog, size_t team) {
  int best = 1;
  size_t most = 0;
  for (int t = std::min(4, groups); t >= 1; --t) {
    const size_t resident = std::min<size_t>(kSmemLimit / (prog + t * team + 1024), 32) * t;
    if (resident > most) {
      most = resident;
      best = t;
    }
  }
  return best;
}

template <typename T, int V, int LS, int TW>
void launch_tasks(const TaskStage& st, const FactorArgs<T, T>& a, const int* meta, const int* words, int lanes,
                  cudaStream_t s) {
  using Team = TaskTeam<T, V, LS, TW>;
  const int groups = (lanes + Team::S - 1) / Team::S;
  const size_t prog = (size_t)(st.max_words + 3) / 4 * 16;
  const size_t team = (size_t)(st.max_arena + 8) * Team::S * sizeof(T);
  int teams = 1;
  if (TW == 1) teams = teams_per_block(groups, prog, team);
  const int blocks_per_task = (groups + teams - 1) / teams;
  const size_t smem = prog + teams * team;
  if (smem > kSmemLimit) throw std::runtime_error("factor tasks: a task exceeds shared memory");
  auto kern = k_factor_tasks<T, V, LS, TW>;
  allow_full_smem(reinterpret_cast<const void*>(kern));
  launch_chained(kern, dim3((unsigned)(st.count * blocks_per_task)), dim3(TW == 1 ? teams * 32 : TW * 32), smem, s,
                 "factor tasks", a, meta + 4 * (size_t)st.begin, words, groups, blocks_per_task, (int)prog,
                 st.max_arena);
}

template <typename T>
void launch_factor_stage(const TaskStage& st, const FactorArgs<T, T>& a, const int* meta, const int* words, int lanes,
                         cudaStream_t s) {
  if (lanes == 1) {  // a single system: every thread a worker
    if (st.warps > 1) launch_tasks<T, 1, 1, 4>(st, a, meta, words, lanes, s);
    else launch_tasks<T, 1, 1, 1>(st, a, meta, words, lanes, s);
    return;
  }
  const auto is = [&](int warps, int lanes_, int pack) {
    return st.warps == warps && st.lanes == lanes_ && st.pack == pack;
  };
  constexpr int kTopLanes = sizeof(T) == 8 ? 4 : 8;
  // the shapes factor_task_specs uses; any other would leave its fronts unfactored
  if (is(1, 8, 1)) return launch_tasks<T, 1, 8, 1>(st, a, meta, words, lanes, s);
  if (is(1, 8, 2)) return launch_tasks<T, 2, 8, 1>(st, a, meta, words, lanes, s);
  if (is(2, 8, 1)) return launch_tasks<T, 1, 8, 2>(st, a, meta, words, lanes, s);
  if (is(4, 8, 1)) return launch_tasks<T, 1, 8, 4>(st, a, meta, words, lanes, s);
  if (is(8, kTopLanes, 1)) return launch_tasks<T, 1, kTopLanes, 8>(st, a, meta, words, lanes, s);
  if constexpr (sizeof(T) == 4) {
    if (is(1, 8, 4)) return launch_tasks<T, 4, 8, 1>(st, a, meta, words, lanes, s);
    if (is(2, 8, 2)) return launch_tasks<T, 2, 8, 2>(st, a, meta, words, lanes, s);
  }
  throw std::runtime_error("factor tasks: no kernel for teams of " + std::to_string(st.warps) + " warps, " +
                           std::to_string(st.lanes) + " lanes, " + std::to_string(st.pack) + " scenarios a lane");
}

}  // namespace cupf_b200
