// task_plan.cpp -- see task_plan.hpp.
#include "task_plan.hpp"

#include <algorithm>
#include <cstring>
#include <limits>

namespace cupf_b200 {
namespace {

// First-fit placement of the arrays of a task in its arena.
struct Arena {
  struct Block {
    int at, size;
  };
  std::vector<Block> used;  // ascending
  int peak = 0;
  int alloc(int size) {
    int at = 0;
    size_t k = 0;
    for (; k < used.size(); ++k) {
      if (used[k].at - at >= size) break;
      at = used[k].at + used[k].size;
    }
    used.insert(used.begin() + k, {at, size});
    peak = std::max(peak, at + size);
    return at;
  }
  void release(int at) {
    for (size_t k = 0; k < used.size(); ++k)
      if (used[k].at == at) {
        used.erase(used.begin() + k);
        return;
      }
  }
};

struct Shared {
  const FactorProgram& fp;
  std::vector<std::vector<int32_t>> kids;  // children, ascending
  std::vector<double> work;                // of one front
  std::vector<uint8_t> done;               // factored by an earlier stage
  std::vector<int32_t> pos;                // position in the task being built, -1 outside it
};

// The fronts below and including the roots that no earlier stage took, children
// before parents; the larger subtrees first, so that few contribution blocks
// wait for their parent at a time.
std::vector<int32_t> task_order(const Shared& sh, const std::vector<int32_t>& roots) {
  std::vector<int32_t> order;
  for (const int32_t root : roots) {
    std::vector<std::pair<int32_t, size_t>> st;
    std::vector<std::vector<int32_t>> todo;
    auto push = [&](int32_t p) {
      std::vector<int32_t> c;
      for (int32_t k : sh.kids[p])
        if (!sh.done[k]) c.push_back(k);
      std::stable_sort(c.begin(), c.end(), [&](int32_t a, int32_t b) { return sh.fp.fsz[a] > sh.fp.fsz[b]; });
      st.push_back({p, 0});
      todo.push_back(c);
    };
    push(root);
    while (!st.empty()) {
      auto& [p, k] = st.back();
      if (k < todo.back().size()) {
        const int32_t c = todo.back()[k++];
        push(c);
      } else {
        order.push_back(p);
        st.pop_back();
        todo.pop_back();
      }
    }
  }
  return order;
}

// Lists of one front.
struct FrontLists {
  std::vector<int32_t> jsrc, jdst, zdst, dst;
  std::vector<std::vector<int32_t>> pass;  // source arena elements, pass by pass
  std::vector<int32_t> ext;                // global CB element, elements, arena element
};

struct TaskBuild {
  std::vector<int32_t> words;
  int arena = 0, fronts = 0;
};

// The task of the fronts below and including the roots that no earlier stage
// factored; false when it exceeds the spec's limits.
bool build_task(Shared& sh, const std::vector<int32_t>& roots, const TaskStageSpec& spec, TaskBuild* out) {
  const FactorProgram& fp = sh.fp;
  const std::vector<int32_t> order = task_order(sh, roots);
  const auto is_root = [&](int32_t p) { return std::find(roots.begin(), roots.end(), p) != roots.end(); };
  const size_t n = order.size();
  std::vector<int> f_at(n), cb_at(n, -1);
  std::vector<std::vector<int>> ext_at(n);
  std::vector<int32_t>& pos = sh.pos;
  for (size_t i = 0; i < n; ++i) pos[order[i]] = (int32_t)i;
  struct Reset {
    std::vector<int32_t>& pos;
    const std::vector<int32_t>& order;
    ~Reset() {
      for (int32_t p : order) pos[p] = -1;
    }
  } reset{pos, order};
  auto cb_size = [&](int32_t p) {
    const int uc = fp.fsz[p] - fp.nc[p];
    return uc * (uc + 1);
  };
  Arena ar;
  auto fetch = [&](size_t i) {  // what the prefetch of front i fills
    const int32_t p = order[i];
    f_at[i] = ar.alloc(fp.fsz[p] * task_front_stride(fp.fsz[p]));
    for (int32_t c : sh.kids[p])
      if (pos[c] < 0 && cb_size(c) > 0) ext_at[i].push_back(ar.alloc(cb_size(c)));
  };
  std::vector<std::vector<int>> src_at(n);  // per child of order[i], its block's arena element (-1: empty)
  fetch(0);
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    size_t e = 0;
    for (int32_t c : sh.kids[p]) {
      int at = -1;
      if (cb_size(c) > 0) at = pos[c] < 0 ? ext_at[i][e++] : cb_at[pos[c]];
      src_at[i].push_back(at);
    }
    for (int at : src_at[i])
      if (at >= 0) ar.release(at);
    if (i + 1 < n) fetch(i + 1);
    if (!is_root(p) && cb_size(p) > 0) cb_at[i] = ar.alloc(cb_size(p));
    ar.release(f_at[i]);
  }
  if (ar.peak > spec.arena_cap || ar.peak > 0xffff) return false;
  out->arena = ar.peak;
  out->fronts = (int)n;
  // programs
  std::vector<int32_t>& w = out->words;
  w.clear();
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    const int fs = fp.fsz[p], nc = fp.nc[p], rs = task_front_stride(fs);
    FrontLists l;
    std::vector<uint8_t> set((size_t)fs * (fs + 1), 0);
    for (int r = 0; r < fs; ++r)
      for (int32_t a = fp.arow_ptr[fp.front_ptr[p] + r]; a < fp.arow_ptr[fp.front_ptr[p] + r + 1]; ++a) {
        l.jsrc.push_back(fp.arow_q[a]);
        l.jdst.push_back(r * rs + fp.arow_col[a]);
        set[(size_t)r * (fs + 1) + fp.arow_col[a]] = 1;
      }
    for (int k = 0; k < nc; ++k) set[(size_t)k * (fs + 1) + fs] = 1;  // the right-hand side rows
    for (int r = 0; r < fs; ++r)
      for (int c = 0; c <= fs; ++c)
        if (!set[(size_t)r * (fs + 1) + c]) l.zdst.push_back(r * rs + c);
    // child terms per destination, children ascending (the order of every
    // other assembly of the engine), destinations by falling term count
    std::vector<std::vector<int32_t>> terms((size_t)fs * (fs + 1));
    for (size_t ci = 0; ci < sh.kids[p].size(); ++ci) {
      const int32_t c = sh.kids[p][ci];
      const int ucc = fp.fsz[c] - fp.nc[c];
      if (ucc == 0) continue;
      const int at = src_at[i][ci];
      if (pos[c] < 0) {
        l.ext.push_back((int32_t)fp.cb_off[c]);
        l.ext.push_back(ucc * (ucc + 1));
        l.ext.push_back(at);
      }
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int r = 0; r < ucc; ++r)
        for (int cc = 0; cc <= ucc; ++cc)
          terms[(size_t)al[r] * (fs + 1) + (cc < ucc ? al[cc] : fs)].push_back(at + r * (ucc + 1) + cc);
    }
    std::vector<int32_t> slots;
    for (int s = 0; s < fs * (fs + 1); ++s)
      if (!terms[s].empty()) slots.push_back(s);
    std::stable_sort(slots.begin(), slots.end(), [&](int32_t a, int32_t b) { return terms[a].size() > terms[b].size(); });
    const size_t npass = slots.empty() ? 0 : terms[slots[0]].size();
    l.pass.resize(npass);
    for (int32_t s : slots) {
      l.dst.push_back(s / (fs + 1) * rs + s % (fs + 1));
      for (size_t k = 0; k < terms[s].size(); ++k) l.pass[k].push_back(terms[s][k]);
    }
    const size_t at = w.size();
    w.resize(at + kTaskRecordWords, 0);
    w[at + kTwShape] = fs | nc << 8 | (is_root(p) ? 1 : 0) << 16;
    w[at + kTwFirst] = fp.first[p];
    w[at + kTwU] = (int32_t)fp.u_off[p];
    w[at + kTwL] = (int32_t)fp.l_off[p];
    w[at + kTwCb] = (int32_t)fp.cb_off[p];
    w[at + kTwFront] = f_at[i];
    w[at + kTwCbArena] = cb_at[i];
    w[at + kTwJ] = (int32_t)(l.jsrc.size() | l.zdst.size() << 16);
    w[at + kTwPass] = (int32_t)npass;
    w[at + kTwExt] = (int32_t)(l.ext.size() / 3);
    for (const auto& q : l.pass) w.push_back((int32_t)q.size());
    w.insert(w.end(), l.ext.begin(), l.ext.end());
    w.insert(w.end(), l.jsrc.begin(), l.jsrc.end());
    for (const auto& q : l.pass)
      for (size_t k = 0; k < q.size(); ++k) w.push_back((int32_t)((uint32_t)l.dst[k] | (uint32_t)q[k] << 16));
    w[at + kTwHalf] = (int32_t)(w.size() - at);
    std::vector<uint16_t> h;
    auto put = [&](const std::vector<int32_t>& v) {
      for (int32_t x : v) h.push_back((uint16_t)x);
    };
    put(l.jdst);
    put(l.zdst);
    if (h.size() % 2) h.push_back(0);
    const size_t hw = w.size();
    w.resize(hw + h.size() / 2);
    if (!h.empty()) std::memcpy(w.data() + hw, h.data(), h.size() * sizeof(uint16_t));
    w[at + kTwNext] = (int32_t)(w.size() - at);
    if ((int)w.size() > spec.word_cap) return false;
  }
  while (w.size() % 4) w.push_back(0);
  return (int)w.size() <= spec.word_cap;
}

// Cuts the tree into stages of tasks.  out marks the fronts to leave out
// (closed towards the root); build(roots, spec) makes one task or says that it
// does not fit; stage(tasks, spec) takes a finished stage, heaviest first.
template <typename Task, typename Build, typename Stage>
void cut_tree(Shared& sh, std::vector<uint8_t>& out, const std::vector<TaskStageSpec>& specs, Build build, Stage stage) {
  const FactorProgram& fp = sh.fp;
  struct Made {
    double work;
    std::vector<int32_t> roots;
    Task t;
  };
  std::vector<double> sub(fp.P);
  for (size_t round = 0;; ++round) {
    const TaskStageSpec& spec = specs[std::min(round, specs.size() - 1)];
    const bool last = round + 1 >= specs.size();
    int32_t left = 0;
    for (int32_t p = 0; p < fp.P; ++p) {
      if (sh.done[p] || out[p]) continue;
      ++left;
      sub[p] = sh.work[p];
      for (int32_t c : sh.kids[p])
        if (!sh.done[c]) sub[p] += sub[c];
    }
    if (!left) return;
    // roots: maximal subtrees of what is left within the cut, split further
    // where one exceeds the spec's limits
    const double cut = spec.cut > 0 && !last ? spec.cut : std::numeric_limits<double>::infinity();
    std::vector<Made> made;
    std::vector<int32_t> todo;
    for (int32_t p = 0; p < fp.P; ++p) {
      if (sh.done[p] || out[p]) continue;
      const int32_t par = fp.parent_panel[p];
      if (par < 0 || out[par]) todo.push_back(p);
    }
    bool dropped = false;
    while (!todo.empty()) {
      const int32_t p = todo.back();
      todo.pop_back();
      Made m{sub[p], {p}, {}};
      if (sub[p] <= cut && build(m.roots, spec, &m.t)) {
        made.push_back(std::move(m));
        continue;
      }
      bool any = false;
      for (int32_t c : sh.kids[p])
        if (!sh.done[c]) {
          todo.push_back(c);
          any = true;
        }
      if (!any && last) {  // does not fit alone: left out with its ancestors
        for (int32_t q = p; q >= 0 && !out[q]; q = fp.parent_panel[q]) out[q] = 1;
        dropped = true;
      }
    }
    if (made.empty()) {
      if (last && !dropped) return;
      continue;
    }
    const auto heavier = [](const Made& a, const Made& b) { return a.work > b.work; };
    std::stable_sort(made.begin(), made.end(), heavier);
    if (spec.merge > 0) {  // small subtrees share a task: fewer starts, longer pipelines
      std::vector<Made> joined;
      size_t lo = 0, hi = made.size();  // [lo, hi) not joined yet: a heavy one takes light ones
      while (lo < hi) {
        Made m = std::move(made[lo++]);
        while (lo < hi && m.work + made[hi - 1].work <= spec.merge) {
          std::vector<int32_t> roots = m.roots;
          roots.insert(roots.end(), made[hi - 1].roots.begin(), made[hi - 1].roots.end());
          Task t{};
          if (!build(roots, spec, &t)) break;
          m.work += made[--hi].work;
          m.roots = std::move(roots);
          m.t = std::move(t);
        }
        joined.push_back(std::move(m));
      }
      made = std::move(joined);
      std::stable_sort(made.begin(), made.end(), heavier);
    }
    for (const Made& m : made) {
      std::vector<int32_t> stack = m.roots;
      while (!stack.empty()) {
        const int32_t q = stack.back();
        stack.pop_back();
        sh.done[q] = 1;
        for (int32_t c : sh.kids[q])
          if (!sh.done[c]) stack.push_back(c);
      }
    }
    std::vector<Task> tasks;
    for (Made& m : made) tasks.push_back(std::move(m.t));
    stage(tasks, spec);
  }
}

// Children and parents of the tree; false when it is not one this code cuts.
bool link_tree(const FactorProgram& fp, Shared* sh) {
  sh->kids.resize(fp.P);
  sh->work.resize(fp.P);
  sh->done.assign(fp.P, 0);
  for (int32_t p = 0; p < fp.P; ++p) {
    const int32_t par = fp.parent_panel[p];
    if (par >= 0 && par <= p) return false;
    if (par >= 0) sh->kids[par].push_back(p);
  }
  return true;
}

struct SweepBuild {
  std::vector<int32_t> words;
  int fronts = 0, ext_rows = 0, local = 0, arena = 0, rows = 0, max_u = 0, max_l = 0;
};

bool build_sweep_task(Shared& sh, const std::vector<int32_t>& roots, const TaskStageSpec& spec, const std::vector<int64_t>& tv_off,
                      const std::vector<int32_t>& level_counts, SweepBuild* out) {
  const FactorProgram& fp = sh.fp;
  const std::vector<int32_t> order = task_order(sh, roots);
  const size_t n = order.size();
  const auto ucof = [&](int32_t p) { return fp.fsz[p] - fp.nc[p]; };
  const auto is_root = [&](int32_t p) { return std::find(roots.begin(), roots.end(), p) != roots.end(); };
  // local numbers: the task's pivots, then the roots' contribution rows
  int npiv = 0;
  for (int32_t p : order) npiv += fp.nc[p];
  std::vector<int32_t> ext_rows;
  for (int32_t r : roots)
    ext_rows.insert(ext_rows.end(), fp.front_rows.begin() + fp.front_ptr[r] + fp.nc[r],
                    fp.front_rows.begin() + fp.front_ptr[r + 1]);
  std::sort(ext_rows.begin(), ext_rows.end());
  ext_rows.erase(std::unique(ext_rows.begin(), ext_rows.end()), ext_rows.end());
  out->local = npiv + (int)ext_rows.size();
  out->ext_rows = (int)ext_rows.size();
  out->fronts = (int)n;
  if (out->local > spec.arena_cap || out->local > 0xffff) return false;
  std::vector<int32_t>& pos = sh.pos;
  for (size_t i = 0; i < n; ++i) pos[order[i]] = (int32_t)i;
  struct Reset {
    std::vector<int32_t>& pos;
    const std::vector<int32_t>& order;
    ~Reset() {
      for (int32_t p : order) pos[p] = -1;
    }
  } reset{pos, order};
  std::vector<int> lp(n), tv_at(n, -1);
  std::vector<std::pair<int32_t, int>> local;  // global pivot row -> local number
  int at = 0;
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    lp[i] = at;
    for (int k = 0; k < fp.nc[p]; ++k) local.push_back({fp.first[p] + k, at++});
  }
  for (int32_t row : ext_rows) local.push_back({row, at++});
  std::sort(local.begin(), local.end());
  const auto number = [&](int32_t row) {
    const auto it = std::lower_bound(local.begin(), local.end(), std::make_pair(row, -1));
    return it != local.end() && it->first == row ? it->second : -1;
  };
  // update vectors in the arena: a front's external children are fetched with
  // its factors, sweep_ring - 1 fronts ahead
  Arena ar;
  std::vector<std::vector<int>> ext_at(n), src_at(n);
  const auto fetch = [&](size_t i) {
    for (int32_t c : sh.kids[order[i]])
      if (pos[c] < 0 && ucof(c) > 0) ext_at[i].push_back(ar.alloc(ucof(c)));
  };
  const size_t ahead = (size_t)sweep_ring(spec.warps) - 1;
  for (size_t i = 0; i < std::min(ahead, n); ++i) fetch(i);
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    size_t e = 0;
    for (int32_t c : sh.kids[p]) src_at[i].push_back(ucof(c) == 0 ? -1 : pos[c] < 0 ? ext_at[i][e++] : tv_at[pos[c]]);
    for (int a : src_at[i])
      if (a >= 0) ar.release(a);
    if (i + ahead < n) fetch(i + ahead);
    if (!is_root(p) && ucof(p) > 0) tv_at[i] = ar.alloc(ucof(p));
  }
  out->arena = ar.peak;
  if (ar.peak > spec.arena_cap || ar.peak > 0xffff) return false;
  std::vector<int32_t>& w = out->words;
  w.assign(n, 0);
  w.insert(w.end(), ext_rows.begin(), ext_rows.end());
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    const int fs = fp.fsz[p], nc = fp.nc[p], uc = fs - nc;
    const size_t r = w.size();
    w[i] = (int32_t)r;
    out->rows = std::max(out->rows, fs);
    out->max_u = std::max(out->max_u, nc * fs);
    out->max_l = std::max(out->max_l, uc * nc);
    if (nc * fs > spec.factor_cap || 64 + uc * nc > spec.factor_cap || fs > spec.factor_cap) return false;
    std::vector<std::vector<int32_t>> terms(fs);
    std::vector<int32_t> ext;
    for (size_t ci = 0; ci < sh.kids[p].size(); ++ci) {
      const int32_t c = sh.kids[p][ci];
      if (ucof(c) == 0) continue;
      if (pos[c] < 0) ext.insert(ext.end(), {(int32_t)tv_off[c], ucof(c), src_at[i][ci]});
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int q = 0; q < ucof(c); ++q) terms[al[q]].push_back(src_at[i][ci] + q);
    }
    std::vector<int32_t> rows;
    for (int q = 0; q < fs; ++q) rows.push_back(q);  // (rows without terms come last and start at zero)
    std::stable_sort(rows.begin(), rows.end(), [&](int32_t a, int32_t b) { return terms[a].size() > terms[b].size(); });
    const size_t npass = terms[rows[0]].size();
    std::vector<std::vector<int32_t>> pass(npass);
    for (int32_t q : rows)
      for (size_t k = 0; k < terms[q].size(); ++k) pass[k].push_back(terms[q][k]);
    w.resize(r + kSweepRecordWords, 0);
    w[r + kSwShape] = fs | nc << 16;
    w[r + kSwFirst] = fp.first[p];
    w[r + kSwU] = (int32_t)fp.u_off[p];
    w[r + kSwL] = (int32_t)fp.l_off[p];
    w[r + kSwLocal] = lp[i];
    w[r + kSwTv] = (int32_t)tv_off[p];
    w[r + kSwTvArena] = tv_at[i];
    w[r + kSwPass] = (int32_t)npass;
    w[r + kSwExt] = (int32_t)(ext.size() / 3);
    w[r + kSwLevel] = level_counts[p];
    for (const auto& q : pass) w.push_back((int32_t)q.size());
    w.insert(w.end(), ext.begin(), ext.end());
    w[r + kSwLists] = (int32_t)(w.size() - r);
    std::vector<uint16_t> h;
    for (int j = 0; j < uc; ++j) {
      const int num = number(fp.front_rows[fp.front_ptr[p] + nc + j]);
      if (num < 0) return false;
      h.push_back((uint16_t)num);
    }
    for (int32_t q : rows) h.push_back((uint16_t)q);
    for (const auto& q : pass)
      for (int32_t s : q) h.push_back((uint16_t)s);
    if (h.size() % 2) h.push_back(0);
    const size_t hw = w.size();
    w.resize(hw + h.size() / 2);
    if (!h.empty()) std::memcpy(w.data() + hw, h.data(), h.size() * sizeof(uint16_t));
    if ((int)w.size() > spec.word_cap) return false;
  }
  while (w.size() % 4) w.push_back(0);
  return (int)w.size() <= spec.word_cap;
}

}  // namespace

// The more systems a batch has, the more of the tree runs as one-warp teams
// (few instructions per front and scenario, no block barriers) and the more
// scenarios a lane carries; with few systems the stages are short instead (a
// few fronts per team), because each launch lasts as long as its longest
// chain of fronts.  One FP32 factorization of the 2,000-bus grid x 1,024
// takes 293 us (521 us with a launch per level; 408 us when the first stage
// is followed by block teams only), the 10,000-bus grid x 64 209 us (540 us
// per level; 315 us with subtrees of up to 2,500 units first).
int task_class(int fronts, int batch) {
  if (batch == 1) return 0;
  const double work = (double)fronts * batch;
  return work > 800e3 && batch > 256 ? 3 : work > 200e3 && batch > 128 ? 2 : 1;
}

// Arena caps keep the launch within shared memory (227 KB): elements x
// lanes x pack x element size per team, programs of at most 44 KB beside it.
std::vector<TaskStageSpec> factor_task_specs(int cls, int elem_bytes) {
  const bool d = elem_bytes == 8;
  const int w = 4000, W = 11000;
  // cut, merge, arena, words, -, warps, lanes, pack
  const TaskStageSpec top{0, 0, 5500, W, 0, 8, d ? 4 : 8, 1};
  switch (cls) {
    case 0:  // (a single system: every thread a worker, whatever the lanes)
      return {{600, 0, 200, w, 0, 1, 8, 1}, {2500, 0, 400, w, 0, 4, 8, 1}, {8000, 0, 2000, W, 0, 4, 8, 1},
              {0, 0, 5500, W, 0, 4, 8, 1}};
    case 1:
      return {{600, 0, 200, w, 0, 1, 8, 1}, {1800, 0, 400, w, 0, 1, 8, 1}, {5000, 0, 1000, W, 0, 4, 8, 1},
              {15000, 0, d ? 2600 : 5500, W, 0, d ? 4 : 8, 8, 1}, top};
    case 2:
      return {{1000, 1500, 130, w, 0, 1, 8, d ? 1 : 2}, {3000, 0, 250, w, 0, 1, 8, 1}, {9000, 0, 600, w, 0, 2, 8, 1},
              {20000, 0, 2000, W, 0, 4, 8, 1}, top};
    default:
      if (d)
        return {{1000, 2000, 130, w, 0, 1, 8, 2}, {2500, 2500, 220, w, 0, 1, 8, 1}, {6000, 0, 450, w, 0, 1, 8, 1},
                {14000, 0, 1000, W, 0, 2, 8, 1}, top};
      return {{1000, 2000, 130, w, 0, 1, 8, 4}, {3000, 0, 250, w, 0, 1, 8, 2}, {8000, 0, 550, w, 0, 2, 8, 2},
              {14000, 0, 1000, W, 0, 2, 8, 1}, top};
  }
}

// Sweeps: a front is a few hundred cycles, so tasks are longer; much work again
// takes wider groups of scenarios per team and joined subtrees.
std::vector<TaskStageSpec> sweep_task_specs(int cls) {
  // cut, merge, arena, words, factor elements, warps, lanes, pack
  if (cls == 3)
    return {{400, 1200, 60, 4000, 80, 1, 16, 1}, {1500, 1500, 160, 4000, 150, 1, 16, 1},
            {0, 0, 2400, 11000, 640, 2, 8, 1}};
  return {{500, 0, 160, 4000, 150, 1, 8, 1}, {2500, 0, 2400, 11000, 640, 2, 8, 1}, {0, 0, 2400, 11000, 640, 2, 8, 1}};
}

TaskPlan build_task_plan(const FactorProgram& fp, int front_limit, const std::vector<TaskStageSpec>& specs) {
  const TaskPlan none{{}, {}, {}, std::vector<uint8_t>(fp.P, 0)};
  // element offsets and list lengths must fit the program's fields
  if (fp.u_total > INT32_MAX || fp.l_total > INT32_MAX || fp.cb_total > INT32_MAX || specs.empty()) return none;
  front_limit = std::min(front_limit, 128);
  Shared sh{fp, {}, {}, {}, std::vector<int32_t>(fp.P, -1)};
  if (!link_tree(fp, &sh)) return none;
  std::vector<uint8_t> out(fp.P, 0);  // left to the level launches
  for (int32_t p = 0; p < fp.P; ++p) {
    const double fs = fp.fsz[p], nc = fp.nc[p], uc = fs - nc;
    sh.work[p] = 60 + fs * (fs + 1) + uc * (uc + 1) * (2 + nc) / 2;
    for (int32_t fr = fp.front_ptr[p]; fr < fp.front_ptr[p + 1]; ++fr)
      for (int32_t a = fp.arow_ptr[fr] + 1; a < fp.arow_ptr[fr + 1]; ++a)
        if (fp.arow_col[a] == fp.arow_col[a - 1]) return none;
    if (fp.fsz[p] >= front_limit)
      for (int32_t q = p; q >= 0 && !out[q]; q = fp.parent_panel[q]) out[q] = 1;
  }
  TaskPlan tp;
  cut_tree<TaskBuild>(
      sh, out, specs, [&](const std::vector<int32_t>& roots, const TaskStageSpec& spec, TaskBuild* t) {
        return build_task(sh, roots, spec, t);
      },
      [&](const std::vector<TaskBuild>& tasks, const TaskStageSpec& spec) {
        TaskStage st;
        st.begin = tp.tasks();
        st.count = (int)tasks.size();
        st.warps = spec.warps;
        st.lanes = spec.lanes;
        st.pack = spec.pack;
        for (const TaskBuild& t : tasks) {
          tp.meta.insert(tp.meta.end(), {(int32_t)tp.words.size(), (int32_t)t.words.size(), t.fronts, 0});
          tp.words.insert(tp.words.end(), t.words.begin(), t.words.end());
          st.max_words = std::max(st.max_words, (int)t.words.size());
          st.max_arena = std::max(st.max_arena, t.arena);
        }
        tp.stages.push_back(st);
      });
  tp.covered = sh.done;
  return tp;
}

SweepPlan build_sweep_plan(const FactorProgram& fp, const std::vector<TaskStageSpec>& specs,
                           const std::vector<int32_t>& level_counts) {
  if (fp.u_total > INT32_MAX || fp.l_total > INT32_MAX || specs.empty()) return {};
  Shared sh{fp, {}, {}, {}, std::vector<int32_t>(fp.P, -1)};
  if (!link_tree(fp, &sh)) return {};
  std::vector<int64_t> tv(fp.P + 1, 0);
  for (int32_t p = 0; p < fp.P; ++p) {
    tv[p + 1] = tv[p] + (fp.fsz[p] - fp.nc[p]);
    sh.work[p] = 30 + fp.nc[p] * fp.fsz[p];
    if (fp.fsz[p] > 0xffff || fp.nc[p] > 8) return {};
  }
  if (tv[fp.P] > INT32_MAX) return {};
  std::vector<uint8_t> out(fp.P, 0);
  SweepPlan sp;
  cut_tree<SweepBuild>(
      sh, out, specs,
      [&](const std::vector<int32_t>& roots, const TaskStageSpec& spec, SweepBuild* t) {
        return build_sweep_task(sh, roots, spec, tv, level_counts, t);
      },
      [&](const std::vector<SweepBuild>& tasks, const TaskStageSpec& spec) {
        SweepTaskStage st;
        st.begin = sp.tasks();
        st.count = (int)tasks.size();
        st.warps = spec.warps;
        st.lanes = spec.lanes;
        st.pack = spec.pack;
        for (const SweepBuild& t : tasks) {
          sp.meta.insert(sp.meta.end(), {(int32_t)sp.words.size(), (int32_t)t.words.size(), t.fronts, t.ext_rows});
          sp.words.insert(sp.words.end(), t.words.begin(), t.words.end());
          st.max_words = std::max(st.max_words, (int)t.words.size());
          st.max_local = std::max(st.max_local, t.local);
          st.max_arena = std::max(st.max_arena, t.arena);
          st.max_rows = std::max(st.max_rows, t.rows);
          st.max_u = std::max(st.max_u, t.max_u);
          st.max_l = std::max(st.max_l, t.max_l);
        }
        sp.stages.push_back(st);
      });
  for (uint8_t d : sh.done)
    if (!d) return {};  // a front too large for a task
  return sp;
}

}  // namespace cupf_b200
