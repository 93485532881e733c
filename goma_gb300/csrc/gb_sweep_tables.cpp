// Host tables of the line sweeps (gb_sweep.cu): the nodes grouped into lines
// of consecutive neighbours, the lines in an order in which every line comes
// after all lines it depends on, and every node's columns.
#include <algorithm>
#include <numeric>

#include "gb_sweep.h"

namespace gb {

// Relative time of a step to the next node of a line (a value handed over in
// shared memory) and of a dependency on another line (a value published
// through L2): only the order of lines and columns follows from them.
static constexpr float kNearTime = 1.0f, kFarTime = 4.0f;

int build_line_tables(const Layout &L, bool upper, LineTables &T) {
  const int nn = L.num_nodes, Tr = L.energy ? L.dim : -1;
  auto adjacent = [&](int a, int b) {
    const int *p = L.nbr_node.data() + L.nbr_ptr[a], *e = L.nbr_node.data() + L.nbr_ptr[a + 1];
    const int *f = std::lower_bound(p, e, b);
    return f != e && *f == b;
  };
  // lines: maximal runs of consecutive nodes of which each couples with the
  // one before it
  std::vector<int> line_of(nn), first;
  for (int n = 0; n < nn; n++) {
    if (n == 0 || !adjacent(n, n - 1)) first.push_back(n);
    line_of[n] = (int)first.size() - 1;
  }
  const int nl = (int)first.size();
  first.push_back(nn);
  // estimated times and the lines' order.  The lines of the dependencies of a
  // line are before it in node order (after it in the upper sweep), so with
  // key(line) >= the keys of its dependencies a stable sort by key keeps
  // every line after them.
  std::vector<float> time(nn, 0.f), key(nl, 0.f);
  const int step = upper ? -1 : 1;
  float last = 1.f;
  for (int q = 0; q < nn; q++) {
    const int n = upper ? nn - 1 - q : q, l = line_of[n];
    const bool start = upper ? n == first[l + 1] - 1 : n == first[l];
    float t = start ? 0.f : time[n - step] + kNearTime;
    for (int k = L.nbr_ptr[n]; k < L.nbr_ptr[n + 1]; k++) {
      const int m = L.nbr_node[k];
      if (upper ? m <= n : m >= n) continue;
      if (line_of[m] == l) continue;
      t = std::max(t, time[m] + kFarTime);
      key[l] = std::max(key[l], key[line_of[m]]);
    }
    time[n] = t;
    last = std::max(last, t);
    if (start) key[l] = std::max(key[l], t);
  }
  T.width = nn * kNearTime / last;
  std::vector<int> order(nl);
  std::iota(order.begin(), order.end(), 0);
  if (upper) std::reverse(order.begin(), order.end());
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key[a] < key[b]; });
  // sizes, then the tasks (near columns: the previous two nodes of the line)
  struct Node {
    int n, n1, n2, nfar;
    int64_t col, val, task;
  };
  std::vector<Node> nodes((size_t)nn);
  T.lines.resize((size_t)nl);
  int64_t ncol = 0, nval = 0, ntask = 0, at = 0;
  for (int l = 0; l < nl; l++) {
    const int a = first[order[l]], b = first[order[l] + 1];
    LineEntry &E = T.lines[(size_t)l];
    E.task0 = (int)ntask;
    E.nnode = b - a;
    for (int i = 0; i < b - a; i++, at++) {
      const int n = upper ? b - 1 - i : a + i;
      Node &N = nodes[(size_t)at];
      N.n = n;
      const int nr = L.fu[n + 1] - L.fu[n];
      auto dofs = [&](int m) { return L.fu[m + 1] - L.fu[m]; };
      N.n1 = i >= 1 ? dofs(n - step) : 0;
      N.n2 = i >= 2 && adjacent(n, n - 2 * step) ? dofs(n - 2 * step) : 0;
      T.wide |= nr > 8;
      N.nfar = nr;  // the node's own right-hand side
      for (int k = L.nbr_ptr[n]; k < L.nbr_ptr[n + 1]; k++) {
        const int m = L.nbr_node[k];
        if (upper ? m <= n : m >= n) continue;
        if ((N.n1 && m == n - step) || (N.n2 && m == n - 2 * step)) continue;
        N.nfar += dofs(m);
      }
      const int nch = (N.nfar + 31) / 32, ng = (nr + 3) / 4;
      if (nch > 65535) return -1;
      N.col = ncol;
      N.val = nval;
      N.task = ntask;
      ncol += nch + 1;
      nval += (int64_t)ng * ((N.n1 + 7) / 8 + (N.n2 + 7) / 8 + 4 * nch);
      ntask += ng;
      if (i == b - a - 1) E.last_nr = nr;
    }
    E.ntask = (int)ntask - E.task0;
  }
  if (ntask > 2147483647LL || ncol > 4294967295LL || nval > 4294967295LL) return -1;
  T.num_groups = nval;
  T.tasks.assign((size_t)ntask, LineTask());
  T.cols.assign((size_t)ncol * 32, kColNone);
  T.src.assign((size_t)ncol * 32, (uint32_t)kColMissing | ((uint32_t)kColMissing << 16));
  std::vector<int> pos_in_line((size_t)nn);
  for (int l = 0, k = 0; l < nl; l++)
    for (int i = 0; i < T.lines[(size_t)l].nnode; i++) pos_in_line[(size_t)k++] = i;
  int bad = 0;
#pragma omp parallel for schedule(dynamic, 256) reduction(| : bad)
  for (int k = 0; k < nn; k++) {
    const Node &N = nodes[(size_t)k];
    const int n = N.n, f0 = L.fu[n], nr = L.fu[n + 1] - f0;
    const int nch = (N.nfar + 31) / 32, ng = (nr + 3) / 4;
    const int n1g = (N.n1 + 7) / 8, n2g = (N.n2 + 7) / 8;
    for (int g = 0; g < ng; g++) {
      LineTask &t = T.tasks[(size_t)(N.task + g)];
      t.val = (uint32_t)(N.val + (int64_t)g * (n1g + n2g + 4 * nch));
      t.col = (uint32_t)N.col;
      t.out = f0 + 4 * g;
      t.nch = (uint16_t)nch;
      t.nrow = (uint8_t)std::min(4, nr - 4 * g);
      t.roff = (uint8_t)(4 * g);
      t.n1 = (uint8_t)N.n1;
      t.n2 = (uint8_t)N.n2;
      t.nr = (uint8_t)nr;
      t.node = pos_in_line[(size_t)k];
      t.id = n;
    }
    int *cols = T.cols.data() + N.col * 32;
    uint32_t *src = T.src.data() + N.col * 32;
    auto put = [&](int64_t p, int slot, int d) {
      const int off = L.nbr_off[slot] + d;
      const int offT = Tr >= 0 && d >= L.nvn ? kColMissing : L.nbr_offT[slot] + d;
      if (off >= kColMissing || (offT >= kColMissing && d < L.nvn)) bad |= 1;
      cols[p] = L.fu[L.nbr_node[slot]] + d;
      src[p] = (uint32_t)(off & 0xffff) | ((uint32_t)(offT & 0xffff) << 16);
    };
    // far columns: the right-hand side, then the neighbours by their time
    int64_t p = 0;
    for (int c = 0; c < nr; c++, p++) {
      cols[p] = kColRhs - c;
      src[p] = (uint32_t)c;
    }
    std::vector<int> far;
    for (int s = L.nbr_ptr[n]; s < L.nbr_ptr[n + 1]; s++) {
      const int m = L.nbr_node[s];
      if (upper ? m <= n : m >= n) continue;
      int near = N.n1 && m == n - step ? 0 : (N.n2 && m == n - 2 * step ? 16 : -1);
      if (near < 0) {
        far.push_back(s);
        continue;
      }
      for (int d = 0; d < L.fu[m + 1] - L.fu[m]; d++) put((int64_t)nch * 32 + near + d, s, d);
    }
    std::stable_sort(far.begin(), far.end(), [&](int a, int b) {
      return time[(size_t)L.nbr_node[a]] < time[(size_t)L.nbr_node[b]];
    });
    for (int s : far)
      for (int d = 0; d < L.fu[L.nbr_node[s] + 1] - L.fu[L.nbr_node[s]]; d++) put(p++, s, d);
  }
  return bad ? -1 : 0;
}

}  // namespace gb
