// Triangular sweeps of the ILU(0) factors by lines of nodes.
//
// What bounds a sweep is its chain of dependencies, not memory: on the 16^3
// HEX27 cube 417 node levels follow one another, and a sweep that hands every
// value over through L2 pays the trip (store, L2, poll) and a block's
// reduction at each of them, 3.3 us a level in FP64.  Most of those levels
// are steps along a line of consecutive nodes: in a mesh numbered line by line
// a Q2 node couples with the two nodes before it, and with nodes of earlier
// lines up to two nodes ahead.  Per element and direction of a 3-D box 18 of
// the 26 levels are such steps.  So a CTA takes a whole line and hands the
// values along it over in shared memory; only the dependencies between lines
// go through L2.
//
// The rows of a node are made independent of one another by scaling: with
// D the node's diagonal block of the factor, the tables hold D^-1 for the
// node's right-hand side and -D^-1 L_nm for every neighbour m before it, so
//     x_n = D^-1 b_n - sum_m (D^-1 L_nm) x_m
// is a sum per row with nothing after it.  (The products D^-1 L_nm are formed
// once per factorisation, in the factors' own type.)  A warp takes up to four
// rows of a node ("task"); the node's columns are one list for all of them.
//   far columns   the right-hand side, then the neighbours outside the line's
//                 last two nodes, oldest first: lane = column, four
//                 accumulators; each value is polled in L2 until published.
//                 The next chunk of 32 columns is on its way while one is
//                 polled and added.
//   near columns  the line's two previous nodes: lane = (column, row); their
//                 values are polled in the shared-memory ring.
// The warps of a CTA take the tasks of its lines in turn, so while one warp
// waits for the node before its own, the others have loaded and summed the
// far columns of the nodes after it.
//
// Order and progress: the CTAs draw lines, one after another, from an order
// in which every line comes after all lines it depends on
// (build_line_tables), and publish their nodes strictly one after another.
// So the lowest unfinished line is always held by a CTA that runs, has all its
// dependencies published and no unfinished line before it: the sweep makes
// progress whatever part of the grid is resident (other streams' kernels may
// hold the rest of the GPU).  The first warp that has no task left in a line draws
// the CTA's next one.  Every wait is bounded: past spin_limit polls a warp
// records an error, goes on with zero and publishes, every later wait stops
// within 1024 polls, and the host reports the failure.
//
// The ring: node i of a CTA's sequence owns slot i mod kRing.  Publication is
// in order, so when a warp starts on a task of node i, its previous task, W
// tasks and so at most W nodes back, is published, and with it every node
// before that task's.  (Other tasks of that node may not be.)  The nodes that
// still read are therefore i-W and later ones: slot i-W-3 has no readers left
// and is set back to the sentinel.  It is polled next for node i-W-3+kRing, by
// a warp working within W of the first unpublished node; that one is past node
// i when kRing > 2W + 2.
//
// All lanes of a warp poll together until none is left waiting: with a loop
// per lane the lanes left it one group at a time and stayed apart, and the
// code after it (six shuffles and adds) took 1,200 clocks instead of 250.
//
// Sums are added in a fixed order: the sweeps are deterministic.
#include <algorithm>
#include <vector>

#include "gb_context.h"
#include "gb_launch.cuh"
#include "gb_publish.cuh"
#include "gb_sweep.h"

namespace gb {

static constexpr unsigned kAll = 0xffffffffu;
static constexpr int kRing = 64;        // nodes in the shared-memory ring
static constexpr int kMaxDofs = 16;     // unknowns per node

// Four rows of one column.  FP64: two 16-byte loads from planes of 32 lanes
// (rows 0-1, then 2-3); FP32: one.
template <class T> struct Rows4 { T r[4]; };
__device__ __forceinline__ Rows4<double> load_rows(const double *v, int lane) {
  const double2 a = __ldcs(reinterpret_cast<const double2 *>(v) + lane);
  const double2 b = __ldcs(reinterpret_cast<const double2 *>(v) + 32 + lane);
  return {{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ Rows4<float> load_rows(const float *v, int lane) {
  const float4 a = __ldcs(reinterpret_cast<const float4 *>(v) + lane);
  return {{a.x, a.y, a.z, a.w}};
}
// position of row r of lane's column within a chunk of 128 values
template <class T>
__device__ __forceinline__ int row_pos(int lane, int r) {
  return sizeof(T) == 4 ? lane * 4 + r : (r >> 1) * 64 + lane * 2 + (r & 1);
}

__device__ __forceinline__ double ld_ring(const double *p) {
  return *reinterpret_cast<const volatile double *>(p);
}
__device__ __forceinline__ float ld_ring(const float *p) {
  return *reinterpret_cast<const volatile float *>(p);
}

__device__ __forceinline__ void st_ring(double *p, double v) {
  *reinterpret_cast<volatile double *>(p) = v;
}
__device__ __forceinline__ void st_ring(float *p, float v) {
  *reinterpret_cast<volatile float *>(p) = v;
}

template <class T>
__global__ void line_gather_kernel(const LineTask *__restrict__ tasks, int64_t ntasks, bool upper,
                                   const int *__restrict__ cols, const uint32_t *__restrict__ src,
                                   LineFactors F, const T *__restrict__ lu,
                                   const T *__restrict__ binv, T *__restrict__ vals) {
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int64_t q = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); q < ntasks;
       q += (int64_t)gridDim.x * wpb) {
    const LineTask t = tasks[q];
    const int f0 = t.out - t.roff, nr = t.nr;
    const T *D = binv + F.inv_ptr[t.id] + (upper ? nr * nr : 0) + t.roff;  // D(r, c) at c * nr + r
    T *v = vals + (size_t)t.val * 32;
    // -sum_k D(r, k) A(k, column) of row r
    auto entry = [&](uint32_t s, int r) -> T {
      const int off = (int)(s & 0xffff), offT = (int)(s >> 16);
      T a = (T)0;
      for (int k = 0; k < nr; k++) {
        const int o = k == F.Tr ? offT : off;
        if (o == kColMissing) continue;
        a = fmx(-D[k * nr + r], lu[F.rowptr[f0 + k] + o], a);
      }
      return a;
    };
    const int64_t cn = ((int64_t)t.col + t.nch) * 32;  // near columns
    for (int h = 0; h < 2; h++) {
      const int n = h ? t.n2 : t.n1;
      for (int c0 = 0; c0 < n; c0 += 8, v += 32) {
        const int c = c0 + (lane >> 2), r = lane & 3;
        v[lane] = c < n && r < t.nrow ? entry(src[cn + 16 * h + c], r) : (T)0;
      }
    }
    for (int k = 0; k < t.nch; k++, v += 128) {
      const int64_t p = ((int64_t)t.col + k) * 32 + lane;
      const int c = cols[p];
      const uint32_t s = src[p];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        T a = (T)0;
        if (c != kColNone && r < t.nrow) a = c < 0 ? D[(int)s * nr + r] : entry(s, r);
        v[row_pos<T>(lane, r)] = a;
      }
    }
  }
}

// The near columns of one earlier node: lane = 4 (column & 1) + row (four
// copies of it in the warp), so a lane holds every other column of its row and
// needs K = 4 products and one exchange.
template <class T, bool WIDE>
struct Near {
  static constexpr int K = WIDE ? 8 : 4;
  T m[K];
  // v: the coefficients, 4 column + row within groups of 8 columns
  __device__ __forceinline__ void load(const T *v, int n, int lane) {
    const int o = lane & 7;  // column parity and row
#pragma unroll
    for (int k = 0; k < K; k++) m[k] = 2 * k < n ? __ldcs(v + 8 * k + o) : (T)0;
  }
  // adds the products with the node's values, lane c holding value c
  __device__ __forceinline__ T add(T x, int n, int lane, T sum) const {
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (2 * k >= n) break;
      const T xc = __shfl_sync(kAll, x, 2 * k + ((lane >> 2) & 1));
      sum = fmx(m[k], xc, sum);
    }
    return sum;
  }
};

template <class T, bool WIDE, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    line_sweep_kernel(LineArgs g, const T *__restrict__ vals, const T *__restrict__ b, T *x) {
  constexpr int W = NT / 32;
  static_assert(2 * W + 2 < kRing, "ring");
  __shared__ T ring[kRing][kMaxDofs];
  // line number k of this CTA: (k << 32) | ticket once drawn
  __shared__ long long drawn[kRing];
  __shared__ int claimed;  // lines drawn or being drawn, less one
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x; k < kRing * kMaxDofs; k += NT) set_unpublished(&ring[0][0] + k);
  if (threadIdx.x < kRing) drawn[threadIdx.x] = -1;
  if (threadIdx.x == 0) claimed = -1;
  dependent_begin();
  __syncthreads();
  const int limit = (int)min(g.spin_limit, 0x7fffffffLL);
  bool gave_up = false;
  int polls = 0;
  auto out_of_polls = [&]() {
    return ++polls > limit || ((polls & 1023) == 0 && *(volatile int *)g.error);
  };
  // this CTA's line number k: drawn by the first warp that needs it
  auto line_of = [&](int k) -> int {
    volatile long long *p = &drawn[k & (kRing - 1)];
    if (lane == 0 && atomicCAS(&claimed, k - 1, k) == k - 1)
      *p = ((long long)k << 32) | (unsigned)atomicAdd(g.ticket, 1);
    __syncwarp();
    long long d = *p;
    while ((int)(d >> 32) != k) {
      if (out_of_polls()) {  // no more lines for this warp; the waits on its nodes run out
        if (lane == 0) atomicExch(g.error, 1);
        return g.nlines;
      }
      d = *p;
    }
    return (int)d;
  };
  // cursor of this warp over the tasks of the CTA's lines: its next task is
  // number pos of line l, the CTA's k-th; base: nodes of the CTA's earlier
  // lines; prev_last: unknowns of the last node of the line before
  int k = 0, l = line_of(0), base = 0, prev_last = 0;
  LineEntry E = l < g.nlines ? g.lines[l] : LineEntry{0, 0, 0, 0};
  for (int pos = threadIdx.x >> 5;; pos += W) {
    while (l < g.nlines && pos >= E.ntask) {
      pos -= E.ntask;
      base += E.nnode;
      prev_last = E.last_nr;
      l = line_of(++k);
      if (l < g.nlines) E = g.lines[l];
    }
    if (l >= g.nlines) break;
    const int4 ta = __ldcs(reinterpret_cast<const int4 *>(g.tasks + E.task0 + pos));
    const int2 tb = __ldcs(reinterpret_cast<const int2 *>(g.tasks + E.task0 + pos) + 2);
    const int out = ta.z, left0 = ta.w & 0xffff, nrow = (ta.w >> 16) & 0xff;
    const int roff = (unsigned)ta.w >> 24, n1 = tb.x & 0xff, n2 = (tb.x >> 8) & 0xff;
    const int node = tb.y, idx = base + node, before = node > 0 ? n1 : prev_last;
    polls = 0;
    gave_up = false;
    const int *cp = g.cols + (size_t)(unsigned)ta.y * 32 + lane;
    int left = left0;
    int c0 = __ldcs(cp), c1 = left > 1 ? __ldcs(cp + 32) : kColNone;
    // slot idx - W - 3 has no readers left (see above)
    if (roff == 0 && idx >= W + 3 && lane < kMaxDofs)
      set_unpublished(&ring[(idx - W - 3) & (kRing - 1)][lane]);
    const T *v = vals + (size_t)(unsigned)ta.x * 32;
    Near<T, WIDE> m1, m2;
    m1.load(v, n1, lane);
    v += 32 * ((n1 + 7) >> 3);
    m2.load(v, n2, lane);
    v += 32 * ((n2 + 7) >> 3);
    const T *rhs = b + (out - roff) + kColRhs;
    auto fetch = [&](int c) -> T {
      const T *p = c >= 0 ? x + c : rhs - c;
      return c != kColNone ? ld_relaxed(p) : (T)0;
    };
    // far columns, a chunk at a time: its values and the next chunk's column
    // and solution value are on their way while it is added
    T s0 = (T)0, s1 = (T)0, s2 = (T)0, s3 = (T)0;
    Rows4<T> a0 = load_rows(v, lane);
    T x0 = fetch(c0);
#pragma unroll 1
    while (true) {
      v += 128;
      cp += 32;
      const int c2 = left > 2 ? __ldcs(cp + 32) : kColNone;
      Rows4<T> a1 = a0;
      if (left > 1) a1 = load_rows(v, lane);
      const T x1 = fetch(c1);
      while (__any_sync(kAll, c0 >= 0 && unpublished(x0))) {
        gave_up |= out_of_polls();
        if (c0 >= 0 && unpublished(x0)) x0 = gave_up ? (T)0 : ld_relaxed(x + c0);
      }
      s0 = fmx(a0.r[0], x0, s0);
      s1 = fmx(a0.r[1], x0, s1);
      if (nrow > 2) {
        s2 = fmx(a0.r[2], x0, s2);
        s3 = fmx(a0.r[3], x0, s3);
      }
      if (--left == 0) break;
      a0 = a1;
      c0 = c1;
      c1 = c2;
      x0 = x1;
    }
    // lane q keeps row q & 3, summed over the warp but for lane q ^ 4
    T sum;
    {
      const bool b0 = lane & 1, b1 = lane & 2;
      const T p0 = (b0 ? s1 : s0) + __shfl_xor_sync(kAll, b0 ? s0 : s1, 1);
      const T p1 = (b0 ? s3 : s2) + __shfl_xor_sync(kAll, b0 ? s2 : s3, 1);
      sum = (b1 ? p1 : p0) + __shfl_xor_sync(kAll, b1 ? p0 : p1, 2);
      sum += __shfl_xor_sync(kAll, sum, 8);
      sum += __shfl_xor_sync(kAll, sum, 16);
    }
    // near columns, the older node first.  At a line's start only the order
    // of publication is waited for.
    auto ring_value = [&](int i, int n) -> T {
      const T *p = &ring[i & (kRing - 1)][lane & (kMaxDofs - 1)];
      T y = lane < n ? ld_ring(p) : (T)0;
      while (__any_sync(kAll, unpublished(y))) {
        gave_up |= out_of_polls();
        if (unpublished(y)) y = gave_up ? (T)0 : ld_ring(p);
      }
      return y;
    };
    T *const slot = &ring[idx & (kRing - 1)][roff + lane];
    T *const xo = x + out + lane;
    if (n2) sum = m2.add(ring_value(idx - 2, n2), n2, lane, sum);
    if (idx > 0) {
      const T x1 = ring_value(idx - 1, before);
      if (node > 0) sum = m1.add(x1, n1, lane, sum);
    }
    sum += __shfl_xor_sync(kAll, sum, 4);
    if (lane < nrow) {
      st_ring(slot, sum);
      st_relaxed(xo, sum);
    }
    if (gave_up && lane == 0) atomicExch(g.error, 1);
  }
}

// ------------------------------------------------------------ host side

template <class V, class D>
static int up(const std::vector<V> &src, D **dst, const char *what) {
  const size_t n = std::max<size_t>(src.size(), 1) * sizeof(V);
  cudaError_t e = cudaMalloc((void **)dst, n);
  if (e == cudaSuccess && !src.empty())
    e = cudaMemcpy(*dst, src.data(), src.size() * sizeof(V), cudaMemcpyHostToDevice);
  return e == cudaSuccess ? 0 : cuda_fail(e, what);
}

int LineSweep::upload(const LineTables &T) {
  nlines = (int)T.lines.size();
  ntasks = (int64_t)T.tasks.size();
  num_groups = T.num_groups;
  wide = T.wide;
  width = T.width;
  std::vector<LineEntry> rev(T.lines.rbegin(), T.lines.rend());
  return up(T.tasks, &d_tasks, "sweep tasks") || up(T.lines, &d_lines, "sweep lines") ||
                 up(rev, &d_lines_rev, "sweep lines") || up(T.cols, &d_cols, "sweep columns") ||
                 up(T.src, &d_src, "sweep columns")
             ? -1
             : 0;
}

void LineSweep::release() {
  void *p[] = {d_tasks, d_lines, d_lines_rev, d_cols, d_src};
  for (void *q : p)
    if (q) cudaFree(q);
  d_tasks = nullptr;
  d_lines = d_lines_rev = nullptr;
  d_cols = nullptr;
  d_src = nullptr;
}

template <class T>
cudaError_t line_gather(const LineSweep &S, bool upper, const LineFactors &F, const T *lu,
                        const T *binv, T *vals, cudaStream_t st) {
  const int grid = (int)std::min<int64_t>((S.ntasks + 7) / 8, 1 << 20);
  line_gather_kernel<T><<<grid, 256, 0, st>>>(S.d_tasks, S.ntasks, upper, S.d_cols, S.d_src, F,
                                              lu, binv, vals);
  return cudaGetLastError();
}

template <class T, bool WIDE, int NT, int MINB>
static cudaError_t launch_lines(const LineArgs &a, const T *vals, const T *b, T *x, int sms,
                                bool one_cta, cudaStream_t st) {
  const int grid = one_cta ? 1 : std::min(a.nlines, MINB * sms);
  launch_dependent(line_sweep_kernel<T, WIDE, NT, MINB>, grid, NT, 0, st, a, vals, b, x);
  return cudaGetLastError();
}

template <class T>
cudaError_t line_sweep(const LineSweep &S, const LineArgs &a, const T *vals, const T *b, T *x,
                       int sms, bool one_cta, cudaStream_t st) {
  LineArgs g = a;
  g.tasks = S.d_tasks;
  g.cols = S.d_cols;
  g.nlines = S.nlines;
  // A line's warps are the nodes it has in work, the CTAs of an SM its lines.
  // Where fewer lines than SMs can run at a time, 16 warps a line and one line
  // an SM; where more can (independent problems, the largest cubes), 12 warps
  // and two lines.  us a sweep, FP64 / FP32:
  //                    lines at a time   16 warps, 1 an SM   12 warps, 2 an SM
  //   16^3 cube                45           317 / 284           372 / 308
  //   24^3 cube                98           510 / 466           592 / 491
  //   32^3 cube               172           911 / 839           836 / 727
  //   16 16^2-32^2 cavities    86           150 / 124           166 / 127
  //   32 of them              172           181 / 157           173 / 140
  //   100 16^2-48^2           400           742 / 561           560 / 409
  const bool many = S.width > sms;
  if (S.wide)
    return many ? launch_lines<T, true, 384, 2>(g, vals, b, x, sms, one_cta, st)
                : launch_lines<T, true, 512, 1>(g, vals, b, x, sms, one_cta, st);
  return many ? launch_lines<T, false, 384, 2>(g, vals, b, x, sms, one_cta, st)
              : launch_lines<T, false, 512, 1>(g, vals, b, x, sms, one_cta, st);
}

template cudaError_t line_gather<double>(const LineSweep &, bool, const LineFactors &,
                                         const double *, const double *, double *, cudaStream_t);
template cudaError_t line_gather<float>(const LineSweep &, bool, const LineFactors &,
                                        const float *, const float *, float *, cudaStream_t);
template cudaError_t line_sweep<double>(const LineSweep &, const LineArgs &, const double *,
                                        const double *, double *, int, bool, cudaStream_t);
template cudaError_t line_sweep<float>(const LineSweep &, const LineArgs &, const float *, const float *,
                                       float *, int, bool, cudaStream_t);

}  // namespace gb
