// Checks the host tables of the line sweeps (gb_sweep_tables.cpp) against the
// layout they were made from; compiled by test_line_tables.py.
#include <cstdio>
#include <cstring>
#include <set>
#include <string>

#include "gb_sweep.h"

using namespace gb;

static std::string check(const Layout &L, bool upper) {
  LineTables T;
  if (build_line_tables(L, upper, T)) return "refused";
  const int nn = L.num_nodes, Tr = L.energy ? L.dim : -1, step = upper ? -1 : 1;
  std::vector<int> node_of(L.N), done(nn, 0), line_of(nn, -1);
  for (int n = 0; n < nn; n++)
    for (int i = L.fu[n]; i < L.fu[n + 1]; i++) node_of[i] = n;
  std::vector<char> used((size_t)T.num_groups, 0);
  int64_t groups = 0;
  size_t next_task = 0;
  for (size_t l = 0; l < T.lines.size(); l++) {
    const LineEntry &E = T.lines[l];
    if ((size_t)E.task0 != next_task || E.ntask <= 0) return "tasks of a line do not follow";
    next_task += E.ntask;
    int node = -1, rows = 0, before[2] = {-1, -1};
    for (int t = E.task0; t < E.task0 + E.ntask; t++) {
      const LineTask &K = T.tasks[t];
      const int n = K.id, f0 = L.fu[n], nr = L.fu[n + 1] - f0;
      if (K.roff == 0) {  // the next node of the line
        if (rows != (node < 0 ? 0 : L.fu[before[0] + 1] - L.fu[before[0]])) return "rows missing";
        if (node >= 0 && n != before[0] + step) return "nodes of a line are not consecutive";
        node++, rows = 0;
        line_of[n] = (int)l;
      }
      if (K.node != node || K.nr != nr || K.out != f0 + K.roff || K.roff != rows || K.nrow < 1 ||
          K.nrow > 4 || K.roff + K.nrow > nr)
        return "a task's rows";
      rows += K.nrow;
      // its values: its own groups, none twice
      const int64_t ng = (K.n1 + 7) / 8 + (K.n2 + 7) / 8 + 4 * (int64_t)K.nch;
      groups += ng;
      for (int64_t g = 0; g < ng; g++) {
        if (K.val + g >= T.num_groups || used[K.val + g]) return "values shared";
        used[K.val + g] = 1;
      }
      if (K.roff) continue;
      // the node's columns: every off-node unknown of the triangle once, the
      // right-hand side once, in the order that the sweep relies on
      std::set<int> want;
      for (int k = L.nbr_ptr[n]; k < L.nbr_ptr[n + 1]; k++) {
        const int m = L.nbr_node[k];
        if (upper ? m <= n : m >= n) continue;
        for (int j = L.fu[m]; j < L.fu[m + 1]; j++) want.insert(j);
      }
      std::set<int> rhs;
      auto entry = [&](int64_t p, int c) -> bool {  // the source of column c
        const int off = T.src[p] & 0xffff, offT = T.src[p] >> 16;
        for (int r = 0; r < nr; r++) {
          const int64_t r0 = L.rowptr[f0 + r], r1 = L.rowptr[f0 + r + 1];
          const int o = r == Tr ? offT : off;
          bool there = false;
          for (int64_t q = r0; q < r1; q++) there |= L.colidx[q] == c;
          if (!there && r == Tr && o == kColMissing) continue;
          if (!there || o == kColMissing || r0 + o >= r1 || L.colidx[r0 + o] != c) return false;
        }
        return true;
      };
      const int64_t far = (int64_t)K.col * 32, near = far + (int64_t)K.nch * 32;
      for (int64_t p = far; p < near; p++) {
        const int c = T.cols[p];
        if (c == kColNone) continue;
        if (c < 0) {
          const int i = kColRhs - c;
          if (i < 0 || i >= nr || (int)T.src[p] != i || !rhs.insert(i).second) return "right-hand side";
          continue;
        }
        const int m = node_of[c];
        if (!want.erase(c)) return "a far column twice or not of the triangle";
        if (line_of[m] < 0 || !done[m]) return "a line before one that it depends on";
        if (!entry(p, c)) return "a far column's entry";
      }
      for (int h = 0; h < 2; h++) {
        const int cnt = h ? K.n2 : K.n1, m = before[h];
        if (cnt && (m < 0 || node <= h || cnt != L.fu[m + 1] - L.fu[m])) return "near columns";
        for (int d = 0; d < cnt; d++) {
          const int64_t p = near + 16 * h + d;
          if (T.cols[p] != L.fu[m] + d || !want.erase(L.fu[m] + d) || !entry(p, L.fu[m] + d))
            return "a near column";
        }
      }
      if (!want.empty()) return "a column is missing";
      if ((int)rhs.size() != nr) return "the right-hand side is missing";
      // later nodes of the line may depend on it
      before[1] = before[0];
      before[0] = n;
      done[n] = 1;
    }
    if (rows != L.fu[before[0] + 1] - L.fu[before[0]]) return "rows missing";
    if (E.nnode != node + 1 || E.last_nr != rows) return "a line's entry";
  }
  if (next_task != T.tasks.size()) return "tasks without a line";
  for (int n = 0; n < nn; n++)
    if (!done[n]) return "a node without a line";
  if (groups != T.num_groups) return "groups without a task";
  return "";
}

extern "C" int line_tables_check(const gb_problem_desc *d, int multicoloured, char *msg) {
  Layout L, Lp;
  std::string err;
  if (build_layout(d, L, err)) {
    strcpy(msg, err.c_str());
    return -1;
  }
  const Layout *LP = &L;
  if (multicoloured) {
    std::vector<int> perm, um;
    std::vector<int64_t> vm;
    multicolour_order(L, perm);
    permute_layout(L, perm, Lp, um, vm);
    LP = &Lp;
  }
  for (int upper = 0; upper < 2; upper++) {
    const std::string e = check(*LP, upper != 0);
    if (!e.empty()) {
      snprintf(msg, 200, "%s sweep: %s", upper ? "upper" : "lower", e.c_str());
      return -1;
    }
  }
  return 0;
}
