// Triangular sweeps of the ILU(0) factors by lines of nodes (gb_sweep.cu):
// host tables (gb_sweep_tables.cpp) and their device copies.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "gb_layout.h"

namespace gb {

// One warp's piece of work in a line sweep: up to four rows of one node.
// The scaled factor values of a task are stored as groups of 32: first the
// near columns (8 columns x 4 rows a group: lane = 4 column + row), then the
// far columns in chunks of 32 (4 groups: all four rows of one column a lane).
struct alignas(16) LineTask {
  uint32_t val;        // first value, in groups of 32
  uint32_t col;        // the node's column list, in groups of 32: nch far groups, one near
  int32_t out;         // first unknown of the task's rows
  uint16_t nch;        // chunks of 32 far columns
  uint8_t nrow, roff;  // rows of the task (1..4), the first one's offset in the node
  uint8_t n1, n2;      // unknowns of the line's previous / second previous node that
                       // the node couples with (near columns; 0: none)
  uint8_t nr, pad;     // unknowns of the node
  int32_t node;        // position of the node in its line
  int32_t id;          // the node
};
static_assert(sizeof(LineTask) == 32, "two 16-byte loads a task");

// One line: its first task, its tasks, its nodes, the unknowns of its last node.
struct alignas(16) LineEntry {
  int32_t task0, ntask, nnode, last_nr;
};

// Entries of a node's column list: an unknown (>= 0) whose solution value the
// sweep has to produce first, kColNone (padding), or kColRhs - c for the
// node's own right-hand side c.
constexpr int kColNone = -1, kColRhs = -2;
constexpr int kColMissing = 0xffff;  // no such entry in the energy row

struct LineTables {
  std::vector<LineTask> tasks;
  std::vector<LineEntry> lines;
  std::vector<int> cols;
  // per column: offset of the entry in a row of the node (energy row
  // separately); right-hand-side columns hold their index in the node
  std::vector<uint32_t> src;  // offset | energy-row offset << 16
  int64_t num_groups = 0;     // groups of 32 values
  double width = 0.0;         // lines that can be worked on at a time, on average
  bool wide = false;          // some node has more than 8 unknowns
};

// Tables of the lower (upper = false) or upper sweep of the layout L.
// Returns -1 when the layout is outside the tables' ranges (a row longer
// than 65,534 entries, more than 2^32 groups): the solver refuses it.
int build_line_tables(const Layout &L, bool upper, LineTables &T);

struct LineArgs {
  const LineTask *tasks;
  const LineEntry *lines;
  const int *cols;
  int nlines;
  long long spin_limit;
  int *error;
  int *ticket;  // next line to be drawn, 0 at the start of a sweep
};

// Device copies for one sweep direction.
struct LineSweep {
  LineTask *d_tasks = nullptr;
  LineEntry *d_lines = nullptr, *d_lines_rev = nullptr;
  int *d_cols = nullptr;
  uint32_t *d_src = nullptr;
  int nlines = 0;
  int64_t ntasks = 0, num_groups = 0;
  bool wide = false;
  double width = 0.0;
  int upload(const LineTables &T);
  void release();
};

// Device layout the factors live in, for the gather below.
struct LineFactors {
  const int *fu;
  const int64_t *rowptr;
  const int64_t *inv_ptr;
  int Tr;  // local index of the energy row, -1 without energy
};

// vals[...] = the scaled factors of every task (see gb_sweep.cu)
template <class T>
cudaError_t line_gather(const LineSweep &S, bool upper, const LineFactors &F, const T *lu,
                        const T *binv, T *vals, cudaStream_t st);
// one sweep: b -> x, x filled with the unpublished sentinel beforehand
template <class T>
cudaError_t line_sweep(const LineSweep &S, const LineArgs &a, const T *vals, const T *b, T *x,
                       int sms, bool one_cta, cudaStream_t st);

}  // namespace gb
