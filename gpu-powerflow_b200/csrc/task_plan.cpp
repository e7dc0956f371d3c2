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
  std::vector<std::vector<int32_t>> kids;     // children, ascending
  std::vector<std::vector<int32_t>> by_size;  // the same, larger fronts first
  std::vector<double> work;                   // of one front
  std::vector<int32_t> words;                 // of one front's record, without its external children
  std::vector<uint8_t> done;                  // factored by an earlier stage
  std::vector<int32_t> pos;                   // position in the task being built, -1 outside it
  int ucof(int32_t p) const { return fp.fsz[p] - fp.nc[p]; }
};

// The fronts below and including the roots that no earlier stage took, children
// before parents; the larger subtrees first, so that few contribution blocks
// wait for their parent at a time.  Stops once their records exceed max_words.
std::vector<int32_t> task_order(const Shared& sh, const std::vector<int32_t>& roots, int64_t max_words) {
  std::vector<int32_t> order;
  std::vector<std::pair<int32_t, size_t>> st;
  int64_t words = 0;
  for (const int32_t root : roots) {
    st.push_back({root, 0});
    while (!st.empty()) {
      auto& [p, k] = st.back();
      const std::vector<int32_t>& kids = sh.by_size[p];
      while (k < kids.size() && sh.done[kids[k]]) ++k;
      if (k < kids.size()) {
        const int32_t c = kids[k++];
        st.push_back({c, 0});
      } else {
        order.push_back(p);
        words += sh.words[p];
        if (words > max_words) return order;
        st.pop_back();
      }
    }
  }
  return order;
}

// Marks a task's fronts with their positions while it is looked at.
struct Positions {
  std::vector<int32_t>& pos;
  const std::vector<int32_t>& order;
  Positions(std::vector<int32_t>& p, const std::vector<int32_t>& o) : pos(p), order(o) {
    for (size_t i = 0; i < order.size(); ++i) pos[order[i]] = (int32_t)i;
  }
  ~Positions() {
    for (int32_t p : order) pos[p] = -1;
  }
};

// A task of the factorization: its fronts and where their arrays lie in the arena.
struct TaskBuild {
  std::vector<int32_t> order;
  std::vector<uint8_t> root;                 // per front
  std::vector<int> f_at, cb_at;              // dense front; contribution block (-1: none, or it leaves)
  std::vector<std::vector<int>> src_at;      // per child, its block's arena element (-1: empty)
  int words = 0, arena = 0;
};

// Appends 16-bit lists, padded to whole words.
void put_halves(std::vector<int32_t>& w, std::vector<uint16_t>& h) {
  if (h.size() % 2) h.push_back(0);
  const size_t at = w.size();
  w.resize(at + h.size() / 2);
  if (!h.empty()) std::memcpy(w.data() + at, h.data(), h.size() * sizeof(uint16_t));
}

// Lays out the task of the fronts below and including the roots that no earlier
// stage factored; false when it exceeds the spec's limits.  Most subtrees are
// tried and not taken, so this counts the program's words without writing them.
bool build_task(Shared& sh, const std::vector<int32_t>& roots, const TaskStageSpec& spec, TaskBuild* out) {
  const FactorProgram& fp = sh.fp;
  out->order = task_order(sh, roots, spec.word_cap);
  const std::vector<int32_t>& order = out->order;
  int64_t words = 0;
  for (int32_t p : order) words += sh.words[p];
  if (words > spec.word_cap) return false;
  const size_t n = order.size();
  out->f_at.assign(n, 0);
  out->cb_at.assign(n, -1);
  out->src_at.assign(n, {});
  out->root.assign(n, 0);
  const Positions mark(sh.pos, order);
  const std::vector<int32_t>& pos = sh.pos;
  for (int32_t r : roots) out->root[pos[r]] = 1;
  auto cb_size = [&](int32_t p) { return sh.ucof(p) * (sh.ucof(p) + 1); };
  Arena ar;
  const auto fetch = [&](size_t i) {  // what the prefetch of front i fills
    const int32_t p = order[i];
    out->f_at[i] = ar.alloc(fp.fsz[p] * task_front_stride(fp.fsz[p]));
    for (int32_t c : sh.kids[p]) {
      const bool ext = pos[c] < 0 && cb_size(c) > 0;
      out->src_at[i].push_back(ext ? ar.alloc(cb_size(c)) : -1);
      if (ext) words += 3;
    }
  };
  fetch(0);
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    for (size_t k = 0; k < sh.kids[p].size(); ++k) {
      int& at = out->src_at[i][k];
      const int32_t c = sh.kids[p][k];
      if (pos[c] >= 0) at = out->cb_at[pos[c]];
      if (at >= 0) ar.release(at);
    }
    if (i + 1 < n) fetch(i + 1);
    if (!out->root[i] && cb_size(p) > 0) out->cb_at[i] = ar.alloc(cb_size(p));
    ar.release(out->f_at[i]);
    if (ar.peak > spec.arena_cap || ar.peak > 0xffff || words > spec.word_cap) return false;
  }
  out->words = (int)(words + 3) / 4 * 4;
  out->arena = ar.peak;
  return out->words <= spec.word_cap;
}

// Writes the task's program.
void write_task(Shared& sh, const TaskBuild& t, std::vector<int32_t>& w) {
  const FactorProgram& fp = sh.fp;
  const Positions mark(sh.pos, t.order);
  const size_t begin = w.size();
  std::vector<int32_t> terms, count, slot_of, dst, pass_at;
  std::vector<uint16_t> h;
  std::vector<uint8_t> set;
  for (size_t i = 0; i < t.order.size(); ++i) {
    const int32_t p = t.order[i];
    const int fs = fp.fsz[p], nc = fp.nc[p], rs = task_front_stride(fs), cols = fs + 1;
    const size_t at = w.size();
    w.resize(at + kTaskRecordWords, 0);
    // child terms per destination, children ascending (the order of every
    // other assembly of the engine), destinations by falling term count
    terms.assign((size_t)fs * cols, 0);
    const auto each_term = [&](auto&& f) {
      for (size_t k = 0; k < sh.kids[p].size(); ++k) {
        const int32_t c = sh.kids[p][k];
        const int ucc = sh.ucof(c), from = t.src_at[i][k];
        const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
        for (int r = 0; r < ucc; ++r)
          for (int cc = 0; cc <= ucc; ++cc) f(al[r] * cols + (cc < ucc ? al[cc] : fs), from + r * (ucc + 1) + cc);
      }
    };
    int npass = 0;
    each_term([&](int s, int) { npass = std::max(npass, ++terms[s]); });
    count.assign(npass + 1, 0);  // destinations with more than k terms
    for (int32_t n : terms)
      for (int k = 0; k < n; ++k) ++count[k];
    slot_of.assign(terms.size(), -1);
    dst.clear();
    for (int n = npass; n > 0; --n)
      for (size_t s = 0; s < terms.size(); ++s)
        if (terms[s] == n) {
          slot_of[s] = (int32_t)dst.size();
          dst.push_back((int32_t)s / cols * rs + (int32_t)s % cols);
        }
    w.insert(w.end(), count.begin(), count.begin() + npass);
    int next = 0;
    for (size_t k = 0; k < sh.kids[p].size(); ++k) {
      const int32_t c = sh.kids[p][k];
      if (sh.pos[c] >= 0 || sh.ucof(c) == 0) continue;
      w.insert(w.end(), {(int32_t)fp.cb_off[c], sh.ucof(c) * (sh.ucof(c) + 1), t.src_at[i][k]});
      ++next;
    }
    h.clear();
    set.assign((size_t)fs * cols, 0);
    int nj = 0;
    for (int r = 0; r < fs; ++r)
      for (int32_t a = fp.arow_ptr[fp.front_ptr[p] + r]; a < fp.arow_ptr[fp.front_ptr[p] + r + 1]; ++a, ++nj) {
        w.push_back(fp.arow_q[a]);
        h.push_back((uint16_t)(r * rs + fp.arow_col[a]));
        set[(size_t)r * cols + fp.arow_col[a]] = 1;
      }
    for (int k = 0; k < nc; ++k) set[(size_t)k * cols + fs] = 1;  // the right-hand side rows
    for (int r = 0; r < fs; ++r)
      for (int c = 0; c < cols; ++c)
        if (!set[(size_t)r * cols + c]) h.push_back((uint16_t)(r * rs + c));
    const int nz = (int)h.size() - nj;
    pass_at.assign(1, (int32_t)w.size());
    for (int k = 0; k < npass; ++k) pass_at.push_back(pass_at[k] + count[k]);
    w.resize(pass_at[npass]);
    std::fill(terms.begin(), terms.end(), 0);
    each_term([&](int s, int from) {
      w[pass_at[terms[s]++] + slot_of[s]] = (int32_t)((uint32_t)dst[slot_of[s]] | (uint32_t)from << 16);
    });
    w[at + kTwShape] = fs | nc << 8 | t.root[i] << 16;
    w[at + kTwFirst] = fp.first[p];
    w[at + kTwU] = (int32_t)fp.u_off[p];
    w[at + kTwL] = (int32_t)fp.l_off[p];
    w[at + kTwCb] = (int32_t)fp.cb_off[p];
    w[at + kTwFront] = t.f_at[i];
    w[at + kTwCbArena] = t.cb_at[i];
    w[at + kTwJ] = (int32_t)((uint32_t)nj | (uint32_t)nz << 16);
    w[at + kTwPass] = npass;
    w[at + kTwExt] = next;
    w[at + kTwHalf] = (int32_t)(w.size() - at);
    put_halves(w, h);
    w[at + kTwNext] = (int32_t)(w.size() - at);
  }
  while ((w.size() - begin) % 4) w.push_back(0);
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
  sh->words.resize(fp.P);
  sh->done.assign(fp.P, 0);
  for (int32_t p = 0; p < fp.P; ++p) {
    const int32_t par = fp.parent_panel[p];
    if (par >= 0 && par <= p) return false;
    if (par >= 0) sh->kids[par].push_back(p);
  }
  sh->by_size = sh->kids;
  for (auto& k : sh->by_size)
    std::stable_sort(k.begin(), k.end(), [&](int32_t a, int32_t b) { return fp.fsz[a] > fp.fsz[b]; });
  return true;
}

// A task of the sweeps: its fronts, and where their update vectors lie in the arena.
struct SweepBuild {
  std::vector<int32_t> order, ext_rows;  // ext_rows: the roots' contribution rows
  std::vector<int> tv_at;                // update vector (-1: none, or it leaves)
  std::vector<std::vector<int>> src_at;  // per child, its vector's arena element (-1: empty)
  int local = 0, words = 0, arena = 0, rows = 0, max_u = 0, max_l = 0;
};

// As build_task; the local numbers are the task's pivots, then ext_rows.
bool build_sweep_task(Shared& sh, const std::vector<int32_t>& roots, const TaskStageSpec& spec, SweepBuild* out) {
  const FactorProgram& fp = sh.fp;
  out->order = task_order(sh, roots, spec.word_cap);
  const std::vector<int32_t>& order = out->order;
  const size_t n = order.size();
  int64_t words = (int64_t)n;
  int npiv = 0;
  *out = SweepBuild{std::move(out->order), {}, {}, {}};
  for (int32_t p : order) {
    const int fs = fp.fsz[p], nc = fp.nc[p], uc = fs - nc;
    words += sh.words[p];
    npiv += nc;
    out->rows = std::max(out->rows, fs);
    out->max_u = std::max(out->max_u, nc * fs);
    out->max_l = std::max(out->max_l, uc * nc);
  }
  if (words > spec.word_cap) return false;
  if (out->max_u > spec.factor_cap || 64 + out->max_l > spec.factor_cap || out->rows > spec.factor_cap) return false;
  std::vector<int32_t>& ext = out->ext_rows;
  for (int32_t r : roots)
    ext.insert(ext.end(), fp.front_rows.begin() + fp.front_ptr[r] + fp.nc[r],
               fp.front_rows.begin() + fp.front_ptr[r + 1]);
  std::sort(ext.begin(), ext.end());
  ext.erase(std::unique(ext.begin(), ext.end()), ext.end());
  words += (int64_t)ext.size();
  out->local = npiv + (int)ext.size();
  if (out->local > spec.arena_cap || out->local > 0xffff) return false;
  const Positions mark(sh.pos, order);
  const std::vector<int32_t>& pos = sh.pos;
  std::vector<uint8_t> root(n, 0);
  for (int32_t r : roots) root[pos[r]] = 1;
  // update vectors in the arena: a front's external children are fetched with
  // its factors, sweep_ring - 1 fronts ahead
  Arena ar;
  out->tv_at.assign(n, -1);
  out->src_at.assign(n, {});
  const auto fetch = [&](size_t i) {
    for (int32_t c : sh.kids[order[i]]) {
      const bool e = pos[c] < 0 && sh.ucof(c) > 0;
      out->src_at[i].push_back(e ? ar.alloc(sh.ucof(c)) : -1);
      if (e) words += 3;
    }
  };
  const size_t ahead = (size_t)sweep_ring(spec.warps) - 1;
  for (size_t i = 0; i < std::min(ahead, n); ++i) fetch(i);
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = order[i];
    for (size_t k = 0; k < sh.kids[p].size(); ++k) {
      int& at = out->src_at[i][k];
      const int32_t c = sh.kids[p][k];
      if (pos[c] >= 0) at = out->tv_at[pos[c]];
      if (at >= 0) ar.release(at);
    }
    if (i + ahead < n) fetch(i + ahead);
    if (!root[i] && sh.ucof(p) > 0) out->tv_at[i] = ar.alloc(sh.ucof(p));
    if (ar.peak > spec.arena_cap || ar.peak > 0xffff || words > spec.word_cap) return false;
  }
  out->words = (int)(words + 3) / 4 * 4;
  out->arena = ar.peak;
  return out->words <= spec.word_cap;
}

// Writes the task's program; number: scratch, -1 for every row.  False when a
// front's row is neither a pivot of the task nor a row of its roots.
bool write_sweep_task(Shared& sh, const SweepBuild& t, const std::vector<int64_t>& tv_off,
                      const std::vector<int32_t>& level_counts, std::vector<int32_t>& number,
                      std::vector<int32_t>& w) {
  const FactorProgram& fp = sh.fp;
  const Positions mark(sh.pos, t.order);
  const size_t begin = w.size(), n = t.order.size();
  std::vector<int> lp(n);
  int at = 0;
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = t.order[i];
    lp[i] = at;
    for (int k = 0; k < fp.nc[p]; ++k) number[fp.first[p] + k] = at++;
  }
  for (int32_t row : t.ext_rows) number[row] = at++;
  bool ok = true;
  w.resize(begin + n, 0);
  w.insert(w.end(), t.ext_rows.begin(), t.ext_rows.end());
  std::vector<int32_t> terms, count, slot_of, pass_at;
  std::vector<uint16_t> h, rows;
  for (size_t i = 0; i < n; ++i) {
    const int32_t p = t.order[i];
    const int fs = fp.fsz[p], nc = fp.nc[p], uc = fs - nc;
    const size_t r = w.size();
    w[begin + i] = (int32_t)(r - begin);
    w.resize(r + kSweepRecordWords, 0);
    // child terms per row, children ascending; rows by falling term count
    // (rows without terms come last and start at zero)
    terms.assign(fs, 0);
    int npass = 0;
    for (const int32_t c : sh.kids[p]) {
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int q = 0; q < sh.ucof(c); ++q) npass = std::max(npass, ++terms[al[q]]);
    }
    count.assign(npass + 1, 0);  // rows with more than k terms
    for (int32_t m : terms)
      for (int k = 0; k < m; ++k) ++count[k];
    slot_of.assign(fs, 0);
    rows.clear();
    for (int m = npass; m >= 0; --m)
      for (int q = 0; q < fs; ++q)
        if (terms[q] == m) {
          slot_of[q] = (int32_t)rows.size();
          rows.push_back((uint16_t)q);
        }
    w.insert(w.end(), count.begin(), count.begin() + npass);
    int next = 0;
    for (size_t k = 0; k < sh.kids[p].size(); ++k) {
      const int32_t c = sh.kids[p][k];
      if (sh.pos[c] >= 0 || sh.ucof(c) == 0) continue;
      w.insert(w.end(), {(int32_t)tv_off[c], sh.ucof(c), t.src_at[i][k]});
      ++next;
    }
    w[r + kSwShape] = fs | nc << 16;
    w[r + kSwFirst] = fp.first[p];
    w[r + kSwU] = (int32_t)fp.u_off[p];
    w[r + kSwL] = (int32_t)fp.l_off[p];
    w[r + kSwLocal] = lp[i];
    w[r + kSwTv] = (int32_t)tv_off[p];
    w[r + kSwTvArena] = t.tv_at[i];
    w[r + kSwPass] = npass;
    w[r + kSwExt] = next;
    w[r + kSwLevel] = level_counts[p];
    w[r + kSwLists] = (int32_t)(w.size() - r);
    h.clear();
    for (int j = 0; j < uc; ++j) {
      const int32_t num = number[fp.front_rows[fp.front_ptr[p] + nc + j]];
      ok = ok && num >= 0;
      h.push_back((uint16_t)num);
    }
    h.insert(h.end(), rows.begin(), rows.end());
    pass_at.assign(1, (int32_t)h.size());
    for (int k = 0; k < npass; ++k) pass_at.push_back(pass_at[k] + count[k]);
    h.resize(pass_at[npass]);
    std::fill(terms.begin(), terms.end(), 0);
    for (size_t k = 0; k < sh.kids[p].size(); ++k) {
      const int32_t c = sh.kids[p][k];
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int q = 0; q < sh.ucof(c); ++q)
        h[pass_at[terms[al[q]]++] + slot_of[al[q]]] = (uint16_t)(t.src_at[i][k] + q);
    }
    put_halves(w, h);
  }
  while ((w.size() - begin) % 4) w.push_back(0);
  for (int32_t p : t.order)
    for (int k = 0; k < fp.nc[p]; ++k) number[fp.first[p] + k] = -1;
  for (int32_t row : t.ext_rows) number[row] = -1;
  return ok;
}

// Words of the halves of a record's lists.
int half_words(int64_t halves) { return (int)((halves + 1) / 2); }

}  // namespace

// The more systems a batch has, the more of the tree runs as one-warp teams
// (few instructions per front and scenario, no block barriers) and the more
// scenarios a lane carries; with few systems the stages are short instead (a
// few fronts per team), because each launch lasts as long as its longest
// chain of fronts.  One FP32 factorization of the 2,000-bus grid x 1,024
// takes 293 us (521 us with a launch per level; 408 us when the first stage
// is followed by block teams only), the 10,000-bus grid x 64 209 us (540 us
// per level; 315 us with subtrees of up to 2,500 units first).
//
// The lines stand where the classes cross on grids of 500 to 10,000 buses.  A
// Newton solve of five updates, us, class 1 / 3: FP32 factors 1,000 buses
// x 1,056 (887k fronts x systems) 1,662 / 1,795, x 1,536 (1,290k) 2,153 / 2,052;
// 1,500 x 704 (887k) 1,865 / 1,858; 2,000 x 480 (802k) 1,900 / 2,086, x 768
// (1,290k) 2,449 / 2,333; 10,000 x 160 (1,344k, but only 160 systems)
// 3,075 / 3,280, x 192 3,509 / 3,463.  FP64 2,000 x 416 (699k) 2,371 / 2,226,
// x 288 (484k) 1,975 / 2,059; 1,000 x 832 (699k) 1,920 / 2,123, x 1,536 3,006 /
// 2,932.  Class 2 is ahead only on trees of a few hundred fronts: 500 buses (420
// fronts) x 1,664 (699k) 1,407 / 1,472 and 1,394 in class 2, FP64 1,784 / 1,862
// and 1,724, x 1,184 (497k) 1,510 / 1,623 and 1,507; 700 buses (589) x 1,184 (696k) 1,509 / 1,640 and 1,780.
int task_class(int fronts, int batch, int elem_bytes) {
  if (batch == 1) return 0;
  const double work = (double)fronts * batch;
  if (fronts < 550) return work > 1100e3 ? 3 : work > 550e3 ? 2 : 1;
  return work > (elem_bytes == 8 ? 720e3 : 900e3) && batch > 160 ? 3 : 1;
}

// Solve and transpose solve, us, class 0 / 3: FP32 700 buses x 2,208 (1,298k)
// 647 / 635, x 2,560 (1,505k) 697 / 664; 1,500 x 1,184 (1,492k) 727 / 727; 2,000 x 544
// (914k) 599 / 657, x 896 (1,505k) 738 / 765, x 1,792 (3,011k) 1,189 / 1,089; FP64 500 x 2,144
// (900k) 575 / 627, x 2,624 (1,102k) 753 / 677; 1,000 x 1,312 (1,102k) 769 / 770;
// 2,000 x 544 749 / 813, x 896 1,056 / 1,032.
int sweep_class(int fronts, int batch, int elem_bytes) {
  return (double)fronts * batch > (elem_bytes == 8 ? 1000e3 : 1400e3) && batch > 256 ? 3 : 0;
}

// Each row is a stage: the most work of a subtree it takes (0: what is left),
// the work up to which subtrees share a task, the arena's and the program's
// limits, and the team.  The cuts are steps of two to four in work, so that a
// stage ends with about as many teams as the GPU holds; the last one takes the
// top of the tree with the widest team.  Arena caps of the one-warp stages
// keep several teams resident on an SM; those of the block teams keep the
// launch within shared memory (227 KB): elements x lanes x pack x element size
// per team, programs of at most 44 KB beside it.  The numbers are the fastest
// tried on 2,000 buses x 1 to 1,024 and 10,000 x 64, and nothing finer is
// claimed for them; which class a batch takes is task_class's choice.
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

// Small trees are a few short levels, and the stages' launches cost as much as
// the levels': per graph-mode iteration 94 us by levels and 113 by tasks
// with 100 buses (about 75 fronts) x 64, 127 and 126 with 300 buses (about 250
// fronts), 220 and 185 with 1,000.
//
// With few systems the time goes by what has to happen one after the other,
// not by the work, and a stage with one long task is slower than the levels it
// replaces.  The line for a single system, against the one launch over the
// tree, is fitted (in us) to Newton solves of 214 random grids of 300 to 9,000
// fronts, with a standard deviation of 6 us about it: the rule's choice is within
// 0.4 % of the faster one on average below 1,400 fronts, where tasks
// always lose 2 % (FP32) and 4 % (FP64), up to 26 %.  500 buses (420
// fronts), one FP64 update: 138 us over the tree, 151 us by tasks; 700 buses
// (589 fronts): 177 and 159.  For 2 to 32 systems only a heaviest chain of more
// than about twice the tree's loses to the levels: 480 buses (408 fronts) x 2
// 135 us by levels, 142 by tasks (FP32); 600 (498 fronts) 186 and 158.
bool tasks_pay(const TaskPlan& tp, int fronts, int batch, int elem_bytes) {
  if (fronts < kTaskFronts || tp.stages.empty()) return false;
  if (fronts >= 2500) return true;
  if (batch == 1)
    return 1.3 * tp.chain + 0.002 * tp.chain_work + (elem_bytes == 8 ? 16 : 13) <
           2.2 * tp.path + 0.0083 * tp.path_work + 3.0 * tp.stages.size();
  return !(batch <= 32 && fronts < 1200 && tp.chain_work > 2.15 * tp.path_work);
}

// The same for the sweeps, whose task works one front after the other: about
// 1.5 us each, against 9 us a level; the more systems, the more a level costs.
// Fitted to the same grids: within 0.7 % of the faster choice on average for
// every batch from 1 to 512 systems, where tasks always lose 1 to 5.6 %.  Solve and
// transpose solve, FP32: 480 buses (chain 49, 12 levels) x 2 256 us by levels
// and 331 by tasks, x 2,048 548 and 462; 600 (chain 44, 15 levels) x 2
// 335 and 322.  Trees of fewer than 400 fronts gain only from a batch
// of a thousand (350 buses, 304 fronts, x 512 285 and 332, x 2,048 478 and 431).
bool sweep_tasks_pay(const SweepPlan& sp, int fronts, int levels, int batch, int elem_bytes) {
  if (fronts < kSweepTaskFronts || sp.stages.empty()) return false;
  if (fronts >= 2500) return true;
  const double items = (double)fronts * std::max(batch, 32);
  if (items > 800e3) return true;
  return sp.chain <= 6.4 * levels - 45 + items / (elem_bytes == 8 ? 30e3 : 45e3);
}

TaskPlan build_task_plan(const FactorProgram& fp, int front_limit, const std::vector<TaskStageSpec>& specs) {
  TaskPlan none;
  none.covered.assign(fp.P, 0);
  // element offsets and list lengths must fit the program's fields
  if (fp.u_total > INT32_MAX || fp.l_total > INT32_MAX || fp.cb_total > INT32_MAX || specs.empty()) return none;
  front_limit = std::min(front_limit, 128);
  Shared sh{fp, {}, {}, {}, {}, {}, std::vector<int32_t>(fp.P, -1)};
  if (!link_tree(fp, &sh)) return none;
  std::vector<uint8_t> out(fp.P, 0);  // left to the level launches
  std::vector<int32_t> scratch;
  for (int32_t p = 0; p < fp.P; ++p) {
    if (fp.nc[p] > 8) return none;  // (the kernels' pivot blocks have up to 8 columns)
    const double fs = fp.fsz[p], nc = fp.nc[p], uc = fs - nc;
    sh.work[p] = 60 + fs * (fs + 1) + uc * (uc + 1) * (2 + nc) / 2;
    for (int32_t fr = fp.front_ptr[p]; fr < fp.front_ptr[p + 1]; ++fr)
      for (int32_t a = fp.arow_ptr[fr] + 1; a < fp.arow_ptr[fr + 1]; ++a)
        if (fp.arow_col[a] == fp.arow_col[a - 1]) return none;
    if (fp.fsz[p] >= front_limit) {
      for (int32_t q = p; q >= 0 && !out[q]; q = fp.parent_panel[q]) out[q] = 1;
      continue;
    }
    // words of its record
    std::vector<int32_t>& count = scratch;
    count.assign((size_t)fp.fsz[p] * (fp.fsz[p] + 1), 0);
    int64_t nj = fp.arow_ptr[fp.front_ptr[p + 1]] - fp.arow_ptr[fp.front_ptr[p]], terms = 0;
    int npass = 0;
    for (int32_t c : sh.kids[p]) {
      const int ucc = sh.ucof(c);
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int r = 0; r < ucc; ++r)
        for (int k = 0; k <= ucc; ++k)
          npass = std::max(npass, ++count[(size_t)al[r] * (fp.fsz[p] + 1) + (k < ucc ? al[k] : fp.fsz[p])]);
      terms += (int64_t)ucc * (ucc + 1);
    }
    // (16-bit lists: every element but the right-hand side rows')
    const int64_t words = kTaskRecordWords + npass + nj + terms + half_words((int64_t)count.size() - fp.nc[p]);
    sh.words[p] = (int32_t)std::min<int64_t>(words, INT32_MAX);
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
        // (the heaviest task comes first)
        tp.chain += (int)tasks[0].order.size();
        for (int32_t p : tasks[0].order) tp.chain_work += sh.work[p];
        for (const TaskBuild& t : tasks) {
          tp.meta.insert(tp.meta.end(), {(int32_t)tp.words.size(), t.words, (int32_t)t.order.size(), 0});
          write_task(sh, t, tp.words);
          st.max_words = std::max(st.max_words, t.words);
          st.max_arena = std::max(st.max_arena, t.arena);
        }
        tp.stages.push_back(st);
      });
  tp.covered = sh.done;
  std::vector<int> depth(fp.P, 0);  // paths from the root down
  std::vector<double> work(fp.P, 0.0);
  for (int32_t p = fp.P - 1; p >= 0; --p) {
    const int32_t par = fp.parent_panel[p];
    depth[p] = 1 + (par >= 0 ? depth[par] : 0);
    work[p] = sh.work[p] + (par >= 0 ? work[par] : 0.0);
    tp.path = std::max(tp.path, depth[p]);
    tp.path_work = std::max(tp.path_work, work[p]);
  }
  return tp;
}

SweepPlan build_sweep_plan(const FactorProgram& fp, const std::vector<TaskStageSpec>& specs,
                           const std::vector<int32_t>& level_counts) {
  if (fp.u_total > INT32_MAX || fp.l_total > INT32_MAX || specs.empty()) return {};
  Shared sh{fp, {}, {}, {}, {}, {}, std::vector<int32_t>(fp.P, -1)};
  if (!link_tree(fp, &sh)) return {};
  std::vector<int64_t> tv(fp.P + 1, 0);
  std::vector<int32_t> count, number(fp.dim, -1);
  bool ok = true;
  for (int32_t p = 0; p < fp.P; ++p) {
    tv[p + 1] = tv[p] + (fp.fsz[p] - fp.nc[p]);
    sh.work[p] = 30 + fp.nc[p] * fp.fsz[p];
    if (fp.fsz[p] > 0xffff || fp.nc[p] > 8) return {};
    int64_t terms = 0;
    int npass = 0;
    count.assign(fp.fsz[p], 0);
    for (int32_t c : sh.kids[p]) {
      const int32_t* al = fp.asm_local.data() + fp.asm_ptr[c];
      for (int q = 0; q < sh.ucof(c); ++q) npass = std::max(npass, ++count[al[q]]);
      terms += sh.ucof(c);
    }
    sh.words[p] = kSweepRecordWords + npass + half_words(sh.ucof(p) + fp.fsz[p] + terms);
  }
  if (tv[fp.P] > INT32_MAX) return {};
  std::vector<uint8_t> out(fp.P, 0);
  SweepPlan sp;
  cut_tree<SweepBuild>(
      sh, out, specs,
      [&](const std::vector<int32_t>& roots, const TaskStageSpec& spec, SweepBuild* t) {
        return build_sweep_task(sh, roots, spec, t);
      },
      [&](const std::vector<SweepBuild>& tasks, const TaskStageSpec& spec) {
        SweepTaskStage st;
        st.begin = sp.tasks();
        st.count = (int)tasks.size();
        st.warps = spec.warps;
        st.lanes = spec.lanes;
        st.pack = spec.pack;
        size_t longest = 0;
        for (const SweepBuild& t : tasks) longest = std::max(longest, t.order.size());
        sp.chain += (int)longest;
        for (const SweepBuild& t : tasks) {
          sp.meta.insert(sp.meta.end(), {(int32_t)sp.words.size(), t.words, (int32_t)t.order.size(),
                                         (int32_t)t.ext_rows.size()});
          ok = write_sweep_task(sh, t, tv, level_counts, number, sp.words) && ok;
          st.max_words = std::max(st.max_words, t.words);
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
  if (!ok) return {};
  return sp;
}

}  // namespace cupf_b200
