// task_plan.hpp -- the front tree cut into subtree tasks for the factorization
// (kernels_task.cuh).
//
// A task is a connected piece of the front tree, or several, its fronts in an
// order that puts children before parents.  One team of threads factors a whole task for
// a handful of scenarios, and the contribution blocks between fronts of the
// task stay in the team's shared memory.  Only the blocks that leave a task
// (its roots') go through global memory.  Tasks are grouped into stages, one
// launch each: the tasks of a stage depend only on earlier stages.
#pragma once

#include <cstdint>
#include <vector>

#include "analysis.hpp"

namespace cupf_b200 {

// One front's record in a task's program (int32 words), followed by its lists:
//   pass counts [npass]        fronts' destinations with > p child terms
//   external children [3 n]    global CB element, elements, arena element
//   jsrc [nJ]                  Jacobian entries
//   terms                      pass by pass: front element | source arena element << 16
//   and as uint16, padded to a word in all: jdst [nJ], zdst [nz].
constexpr int kTaskRecordWords = 12;
enum TaskWord : int {
  kTwShape = 0,   // fs | nc << 8 | (a subtree's root: its contribution block leaves the task) << 16
  kTwFirst = 1,   // first pivot row
  kTwU = 2,       // U, L21 and CB element offsets
  kTwL = 3,
  kTwCb = 4,
  kTwFront = 5,   // arena element of the dense front [fs][front_stride(fs)]
  kTwCbArena = 6, // arena element of its contribution block [uc][uc + 1] (when it stays)
  kTwJ = 7,       // nJ | nz << 16
  kTwPass = 8,    // passes of child terms
  kTwExt = 9,     // external children
  kTwNext = 10,   // words of this record with its lists
  kTwHalf = 11,   // word of the uint16 lists
};

// Row stride of a dense front of a task: fs + 1 entries (the last column is
// the right-hand side) rounded up to odd, so that neighbouring rows start in
// different shared-memory banks; 9 for all fronts of up to 8 rows, whose
// elimination is unrolled over the columns with fixed offsets.
constexpr int kSmallFront = 8;
constexpr int task_front_stride(int fs) { return fs <= kSmallFront ? kSmallFront + 1 : (fs + 1) | 1; }

struct TaskStageSpec {
  double cut = 0;      // most work of one subtree (0: no limit)
  double merge = 0;    // subtrees are joined into tasks of up to this much work (0: one each)
  int arena_cap = 0;   // most arena elements (per scenario) of one task
  int word_cap = 0;    // most program words of one task
  int factor_cap = 0;  // sweeps: most factor elements of one front
  int warps = 1;       // warps of a team (more than one: the block is the team)
  int lanes = 8;       // lanes that share out a team's scenarios ...
  int pack = 1;        // ... and scenarios per lane
};

constexpr int kTaskFronts = 300;       // smallest trees that factor (sweep) as tasks: tasks_pay
constexpr int kSweepTaskFronts = 400;

// Classes of batches with stages of their own: 0 a single system; by the
// fronts x systems of a batch, 1 little and 3 much work, 2 in between on small
// trees.  The sweeps have stages of their own for class 0 and 3.
int task_class(int fronts, int batch, int elem_bytes);
int sweep_class(int fronts, int batch, int elem_bytes);
// The stages of a class, for 4- or 8-byte factors.
std::vector<TaskStageSpec> factor_task_specs(int cls, int elem_bytes);
std::vector<TaskStageSpec> sweep_task_specs(int cls);

struct TaskStage {
  int begin = 0, count = 0;         // tasks
  int max_words = 0, max_arena = 0; // largest program and arena of the stage
  int warps = 1, lanes = 8, pack = 1; // of a team
};

struct TaskPlan {
  std::vector<int32_t> meta;     // per task: program offset (words, a multiple of 4), words, fronts, 0
  std::vector<int32_t> words;
  std::vector<TaskStage> stages; // in launch order
  std::vector<uint8_t> covered;  // per panel: 1 when a task factors it
  // What one factorization of few systems has to do one after the other, in
  // fronts and in units of work: the heaviest task of every stage, and for
  // comparison the longest path of the front tree.
  int chain = 0, path = 0;
  double chain_work = 0, path_work = 0;
  int tasks() const { return (int)(meta.size() / 4); }
};

// ---------------------------------------------------------------------------
// Triangular sweeps over subtree tasks.  The forward sweeps (L y = b,
// U^T w = g) run a task's fronts children first: update vectors pass from
// child to parent in the arena.  The backward sweeps (U x = y, L^T z = w) run
// the stages and the fronts the other way round: the solution rows a front
// needs are its ancestors', kept in the task's own numbering (its pivots,
// then the rows of the roots' contribution blocks, fetched at the start).
// A task's program: [offset of each front's record][external rows][records].
// A record is kSweepRecordWords words, then
//   pass counts [npass], external children [3 n]: update element, rows, arena element
// and as uint16, padded to a word in all: the rows' local numbers [uc], the
// front rows by falling number of child terms [fs], then npass lists of source arena elements.
// ---------------------------------------------------------------------------
constexpr int kSweepRecordWords = 12;
enum SweepWord : int {
  kSwShape = 0,  // fs | nc << 16
  kSwFirst = 1,  // first pivot row
  kSwU = 2,      // U and L21 element offsets
  kSwL = 3,
  kSwLocal = 4,  // local number of the first pivot
  kSwTv = 5,     // element of the update vector in the global array (roots)
  kSwTvArena = 6, // ... or in the arena, -1 at a root
  kSwPass = 7,   // passes of the gather
  kSwExt = 8,    // external children
  kSwLists = 9,  // word of the uint16 lists, from the record's start
  kSwLevel = 10, // fronts of the front's level launch (level_counts)
};

// Fronts whose factors a sweep team has in flight or in use.  A block team runs
// where few teams are resident, so that a front's memory latency is covered
// only by the team's own earlier requests.
constexpr int sweep_ring(int warps) { return warps == 1 ? 2 : 4; }

struct SweepTaskStage {
  int begin = 0, count = 0;
  int max_words = 0;  // largest program
  int max_local = 0;  // most local rows (pivots and external rows)
  int max_arena = 0;  // most arena elements of the forward sweeps
  int max_rows = 0;   // most rows of a front
  int max_u = 0;      // most U elements of a front (nc * fs)
  int max_l = 0;      // most L21 elements of a front (uc * nc)
  int warps = 1, lanes = 8, pack = 1;
};

struct SweepPlan {
  std::vector<int32_t> meta;  // per task: program offset (words), words, fronts, external rows
  std::vector<int32_t> words;
  std::vector<SweepTaskStage> stages;  // leaves first
  int chain = 0;  // fronts of the longest task of every stage
  int tasks() const { return (int)(meta.size() / 4); }
};

// Cuts the whole tree; empty when a front exceeds the records' fields.  Spec
// limits: arena_cap is the most local rows and the most arena elements.
// level_counts: per panel, the fronts of its level launch.
SweepPlan build_sweep_plan(const FactorProgram& fp, const std::vector<TaskStageSpec>& specs,
                           const std::vector<int32_t>& level_counts);

// Cuts the tree.  Fronts of at least `front_limit` rows, and all their
// ancestors, are left out (covered = 0).  The last spec is repeated until no
// front that fits it is left; a front that does not fit it alone is left out
// with its ancestors.  A pattern with repeated entries gives an empty plan.
TaskPlan build_task_plan(const FactorProgram& fp, int front_limit, const std::vector<TaskStageSpec>& specs);

// Whether a batch (1, or the batch padded to 32) factors faster by these tasks
// than by the other schedules, and sweeps faster by tasks than level by level.
bool tasks_pay(const TaskPlan& tp, int fronts, int batch, int elem_bytes);
bool sweep_tasks_pay(const SweepPlan& sp, int fronts, int levels, int batch, int elem_bytes);

}  // namespace cupf_b200
