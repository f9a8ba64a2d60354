// Straight-line PTX for one mechanism's evaluations, factorization and
// triangular solves, shared among the warps of a group's team.
//
// Why straight-line code. The table-driven kernels (rosenbrock.cuh) spend
// about 40 integer, address and control instructions around every FP64
// multiply-add decoding their streams. Here the pattern is known when the plan
// is made, so every operand is an immediate offset from one base register and
// the instruction stream is the arithmetic itself: one DFMA per update plus
// its share of the operand loads.
//
// Why teams. A group is one warp's 32 lanes wide, and one warp issues a DFMA
// every 64 cycles on its SM sub-partition whatever the rest of the chip does,
// so a launch of few groups leaves most of the FP64 units idle. A group is
// therefore worked on by a team of 1 to 16 warps (a block), or a cluster of
// such blocks on several SMs, every warp holding the same 32 cells: the
// generated work is cut into tasks (a row, a block of rows by columns, a range
// of reactions), the tasks are scheduled into steps of kSegments segments that
// depend on earlier steps only, and warp w of W runs segments w, w + W, ... of
// a step before the team's barrier. One module serves every team size, and
// since a task is run by one warp with one order of operations, results do not
// depend on the team size.
//
// The factorization: the leading rows are single-row tasks (their elimination
// DAG gives the parallelism); the rows of the trailing dense square are
// blocks of `tile` rows whose multipliers of the leading pivots are one task
// and whose columns in the square are tiles of `tile` columns, one task each:
// a tile's entries live in registers from assembly to store, and every pivot
// contributes the outer product of its multipliers and its U row, loaded once
// per tile (2t loads for up to t^2 independent FMAs). Only structurally
// nonzero products are emitted. The dense square itself is eliminated by a
// loop over its blocks (dense_lu in rosenbrock.cuh), a few kilobytes of code
// for about 60% of the multiply-adds. Every entry receives the updates of the
// row-by-row elimination in ascending pivot order with the same operations
// (fma(-l, u, a); l = a * (1 / pivot); 1 / pivot by an IEEE division), so the
// factors are those of every other variant bit for bit.
//
// The solves: leading rows are single-row tasks, the square's rows lose their
// terms in the leading columns `solve_block` rows at a time, and the square's
// own triangle is a loop (square_triangle in rosenbrock.cuh). Every row sums its
// terms in the order in which their values finish (ascending columns forward,
// descending columns backward), as the plain variant's loops do, so results
// match that variant bit for bit.
#include "codegen.h"

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <functional>
#include <memory>
#include <stdexcept>
#include <utility>
#include <vector>

#include "layout.h"

namespace fo {
namespace {

class Ptx {
 public:
  std::string body;
  int next = 1;      // %d0 is alpha
  int64_t fmas = 0;  // updates of a factorization emitted

  int reg() { return next++; }

  void line(const char* fmt, ...) __attribute__((format(printf, 2, 3))) {
    char buf[160];
    va_list ap;
    va_start(ap, fmt);
    const int len = vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    body.append("\t");
    body.append(buf, (size_t)std::min<int>(len, (int)sizeof(buf) - 1));
    body.append("\n");
  }
  // value of item `item` of this lane's scratch
  int load(int64_t item) {
    const int r = reg();
    line("ld.global.f64 %%d%d, [%%b+%lld];", r, (long long)(item * 256));
    return r;
  }
  void store(int64_t item, int r) { line("st.global.f64 [%%b+%lld], %%d%d;", (long long)(item * 256), r); }
  int neg(int x) {
    const int r = reg();
    line("neg.f64 %%d%d, %%d%d;", r, x);
    return r;
  }
  int fma(int a, int b, int c) {
    const int r = reg();
    line("fma.rn.f64 %%d%d, %%d%d, %%d%d, %%d%d;", r, a, b, c);
    return r;
  }
  int mul(int a, int b) {
    const int r = reg();
    line("mul.rn.f64 %%d%d, %%d%d, %%d%d;", r, a, b);
    return r;
  }
  int add(int a, int b) {
    const int r = reg();
    line("add.rn.f64 %%d%d, %%d%d, %%d%d;", r, a, b);
    return r;
  }
  int sub(int a, int b) {
    const int r = reg();
    line("sub.rn.f64 %%d%d, %%d%d, %%d%d;", r, a, b);
    return r;
  }
  // a * v and a * v + c with an immediate v
  int mul_imm(int a, double v) {
    const int r = reg();
    line("mul.rn.f64 %%d%d, %%d%d, 0d%016llX;", r, a, bits_of(v));
    return r;
  }
  int fma_imm(int a, double v, int c) {
    const int r = reg();
    line("fma.rn.f64 %%d%d, %%d%d, 0d%016llX, %%d%d;", r, a, bits_of(v), c);
    return r;
  }
  static unsigned long long bits_of(double v) {
    unsigned long long bits;
    static_assert(sizeof(bits) == sizeof(v), "");
    std::memcpy(&bits, &v, sizeof(v));
    return bits;
  }
  int constant(double v) {
    const int r = reg();
    line("mov.f64 %%d%d, 0d%016llX;", r, bits_of(v));
    return r;
  }
  int recip(int x) {
    const int r = reg();
    line("div.rn.f64 %%d%d, 0d3FF0000000000000, %%d%d;", r, x);
    return r;
  }
};

using Emit = std::function<void(Ptx&)>;
// One phase: steps[s][g] is what segment g of step s does.
using Phase = std::vector<std::vector<std::vector<Emit>>>;

// One unit of generated work: `after` lists the tasks it reads from.
struct Task {
  std::vector<int> after;
  Emit emit;
};

// Cost of a task in units of one multiply-add: operand loads and stores take
// about a quarter of a DFMA's issue time, a division nine.
int64_t cost_of(const Task& t) {
  Ptx x;
  t.emit(x);
  int64_t c = 0;
  for (size_t at = 0; at < x.body.size(); at = x.body.find('\n', at) + 1) {
    const char* l = x.body.c_str() + at + 1;
    c += !std::strncmp(l, "ld", 2) || !std::strncmp(l, "st", 2) ? 1 : !std::strncmp(l, "div", 3) ? 36
         : !std::strncmp(l, "neg", 3) || !std::strncmp(l, "mov", 3) ? 0 : 4;
  }
  return c / 4 + 1;
}

// Splits tasks (longest first) between the segments that agree with `seg` in
// their low `bit` bits: two halves of like cost, halved again down to single
// segments. A team of 2^m warps gives a warp the segments that agree in m low
// bits, so every team size finds its warps' loads balanced (one long task
// leaves its warp alone with it).
void halve(const std::vector<int>& tasks, const std::vector<int64_t>& cost, int bit, int seg,
           const std::function<void(int, int)>& place) {
  if (tasks.empty()) return;
  if ((1 << bit) >= kSegments || (tasks.size() == 1)) {
    for (int i : tasks) place(i, seg);
    return;
  }
  std::vector<int> half[2];
  int64_t load[2] = {0, 0};
  for (int i : tasks) {
    const int h = load[1] < load[0] ? 1 : 0;
    half[h].push_back(i);
    load[h] += cost[i];
  }
  for (int h = 0; h < 2; ++h) halve(half[h], cost, bit + 1, seg | (h << bit), place);
}

// Tasks into steps of kSegments segments. A step takes every task whose
// inputs are ready, spread over the segments (halve); a task whose
// last inputs are made in one segment of the step follows them there when
// that does not lengthen the step (a short step is lengthened: a barrier and
// the first loads of a step cost about kStepCost), or when it is the only
// task left to run.
Phase schedule(const std::vector<Task>& tasks) {
  constexpr int64_t kStepCost = 48;
  const int n = (int)tasks.size();
  std::vector<int64_t> cost(n);
  std::vector<int> waits(n, 0), step(n, -1), segment(n, -1);
  std::vector<std::vector<int>> before(n);
  for (int i = 0; i < n; ++i) {
    cost[i] = cost_of(tasks[i]);
    waits[i] = (int)tasks[i].after.size();
    for (int a : tasks[i].after) before[a].push_back(i);
  }
  std::vector<int> ready;
  for (int i = 0; i < n; ++i)
    if (!waits[i]) ready.push_back(i);
  Phase out;
  for (int s = 0, done = 0; done < n; ++s) {
    if (ready.empty()) throw std::logic_error("cyclic tasks");
    std::stable_sort(ready.begin(), ready.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<std::vector<int>> seg(kSegments);
    std::vector<int64_t> load(kSegments, 0);
    std::vector<int> placed, next;
    auto place = [&](int i, int g) {
      seg[g].push_back(i);
      load[g] += cost[i];
      step[i] = s;
      segment[i] = g;
      placed.push_back(i);
      ++done;
    };
    halve(ready, cost, 0, 0, place);
    const bool serial = placed.size() < 3;
    const int64_t limit = std::max(*std::max_element(load.begin(), load.end()), kStepCost);
    for (size_t q = 0; q < placed.size(); ++q) {
      std::vector<int> made;
      for (int i : before[placed[q]])
        if (!--waits[i]) made.push_back(i);
      for (int i : made) {
        // in this step if its inputs of this step share a segment
        int g = -1;
        bool one = true;
        for (int a : tasks[i].after)
          if (step[a] == s) {
            if (g >= 0 && segment[a] != g) one = false;
            g = segment[a];
          }
        const bool alone = serial && made.size() == 1 && next.empty() && q + 1 == placed.size();
        if (one && (alone || load[g] + cost[i] <= limit)) place(i, g);
        else next.push_back(i);
      }
    }
    ready = std::move(next);
    out.emplace_back(kSegments);
    for (int g = 0; g < kSegments; ++g)
      for (int i : seg[g]) out.back()[g].push_back(tasks[i].emit);
    while (!out.back().empty() && out.back().back().empty()) out.back().pop_back();
  }
  return out;
}

// A matrix to factor: its filled pattern, where its entries live, and what
// they start from.
struct Matrix {
  int n = 0, d0 = 0;              // rows from d0 on form the dense square
  std::vector<int64_t> item;      // n*n: item of (i, j), or -1
  std::vector<int64_t> start;     // n*n: item of -J(i, j), or -1 (zero)
  std::vector<double> mass;       // the diagonal gains alpha * mass
  std::vector<char> unit;         // rows that are those of the identity
  int64_t at(int i, int j) const { return item[(size_t)i * n + j]; }
};

Matrix full_matrix(const HostTables& t, const GenLayout& gl) {
  Matrix A;
  A.n = t.n;
  A.d0 = gl.d0;
  A.item.assign((size_t)t.n * t.n, -1);
  A.start.assign((size_t)t.n * t.n, -1);
  A.unit.assign(t.n, 0);
  A.mass = t.mass;
  for (int i = 0; i < t.n; ++i)
    for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q) A.item[(size_t)i * t.n + t.lu_col[q]] = gl.lu_item[q];
  for (int i = 0; i < t.n; ++i)
    for (int e = t.j_row_ptr[i]; e < t.j_row_ptr[i + 1]; ++e) A.start[(size_t)i * t.n + t.j_col[e]] = gl.s.negj + e;
  return A;
}

// The projection's matrix diag(M) - J with the differential rows of J
// dropped (alpha = 1): only the algebraic rows have entries off the diagonal,
// so its factors are a small part of the full pattern's, in the same storage.
Matrix projection_matrix(const HostTables& t, const GenLayout& gl) {
  Matrix A;
  A.n = A.d0 = t.n;
  A.item.assign((size_t)t.n * t.n, -1);
  A.start.assign((size_t)t.n * t.n, -1);
  A.unit.assign(t.n, 0);
  A.mass = t.mass;
  std::vector<char> in((size_t)t.n * t.n, 0);
  for (int i = 0; i < t.n; ++i) {
    in[(size_t)i * t.n + i] = 1;
    A.unit[i] = t.mass[i] == 1.0;
    if (t.mass[i] != 0.0) continue;
    for (int e = t.j_row_ptr[i]; e < t.j_row_ptr[i + 1]; ++e) {
      in[(size_t)i * t.n + t.j_col[e]] = 1;
      A.start[(size_t)i * t.n + t.j_col[e]] = gl.s.negj + e;
    }
  }
  for (int k = 0; k < t.n; ++k)
    for (int i = k + 1; i < t.n; ++i)
      if (in[(size_t)i * t.n + k])
        for (int j = k + 1; j < t.n; ++j)
          if (in[(size_t)k * t.n + j]) in[(size_t)i * t.n + j] = 1;
  int64_t o = gl.s.lu;
  for (size_t q = 0; q < in.size(); ++q)
    if (in[q]) A.item[q] = o++;
  return A;
}

// The columns below `limit` of rows that do not eliminate one another (one
// row, or rows whose columns below `limit` all lie left of them): assembly,
// every pivot's updates in ascending order, the multipliers (in place, and of
// one row the reciprocal pivot and its U entries), `width` columns at a time.
void emit_rows(Ptx& x, const Matrix& A, const std::vector<int>& rows, int limit, int width) {
  std::vector<int> cols;
  for (int j = 0; j < limit; ++j)
    for (int i : rows)
      if (A.at(i, j) >= 0) {
        cols.push_back(j);
        break;
      }
  const int m = (int)rows.size();
  for (size_t c0 = 0; c0 < cols.size(); c0 += width) {
    const size_t c1 = std::min(cols.size(), c0 + width);
    const int first = cols[c0], last = cols[c1 - 1];
    std::vector<int> acc((size_t)m * (c1 - c0), -1), nl(m, -1);
    auto at = [&](int r, size_t c) -> int& { return acc[(size_t)r * (c1 - c0) + (c - c0)]; };
    for (int r = 0; r < m; ++r)
      for (size_t c = c0; c < c1; ++c) {
        const int i = rows[r], j = cols[c];
        if (A.at(i, j) < 0) continue;
        const int64_t from = A.start[(size_t)i * A.n + j];
        int v = from >= 0 ? x.load(from) : x.constant(0.0);
        // alpha * 1 is alpha exactly; any other mass takes the product
        if (i == j) v = x.add(v, A.mass[i] == 1.0 ? 0 : x.mul_imm(0, A.mass[i]));
        at(r, c) = v;
      }
    for (size_t ck = 0; ck < cols.size(); ++ck) {
      const int k = cols[ck];
      if (k >= rows[0] || k > last) break;
      const bool here = k >= first;
      std::vector<size_t> to;
      for (size_t c = c0; c < c1; ++c)
        if (cols[c] > k && A.at(k, cols[c]) >= 0) to.push_back(c);
      if (!here && to.empty()) continue;
      const int rk = here && !A.unit[k] ? x.load(A.at(k, k)) : -1;
      for (int r = 0; r < m; ++r) {
        nl[r] = -1;
        if (A.at(rows[r], k) < 0) continue;
        if (here) {
          int& l = at(r, ck);
          if (rk >= 0) l = x.mul(l, rk);   // else the pivot is 1
          x.store(A.at(rows[r], k), l);
          nl[r] = x.neg(l);
        } else {
          nl[r] = x.neg(x.load(A.at(rows[r], k)));
        }
      }
      for (size_t c : to) {
        const int u = x.load(A.at(k, cols[c]));
        for (int r = 0; r < m; ++r)
          if (nl[r] >= 0) {
            if (at(r, c) < 0) throw std::logic_error("fill pattern not closed");
            at(r, c) = x.fma(nl[r], u, at(r, c));
            ++x.fmas;
          }
      }
    }
    for (int r = 0; r < m; ++r)
      for (size_t c = c0; c < c1; ++c) {
        if (at(r, c) < 0 || cols[c] < rows[r]) continue;
        x.store(A.at(rows[r], cols[c]), cols[c] == rows[r] ? x.recip(at(r, c)) : at(r, c));
      }
  }
}

// A tile of the dense square before its own elimination: assembly (structural
// zeros too) and the updates of the pivots before the square.
void emit_tile(Ptx& x, const Matrix& A, const GenLayout& gl, int i0, int i1, int j0, int j1) {
  const int b = j1 - j0;
  std::vector<int> acc((size_t)(i1 - i0) * b), nl(i1 - i0);
  for (int i = i0; i < i1; ++i)
    for (int j = j0; j < j1; ++j) {
      const int64_t from = A.start[(size_t)i * A.n + j];
      int v = from >= 0 ? x.load(from) : x.constant(0.0);
      if (i == j) v = x.add(v, A.mass[i] == 1.0 ? 0 : x.mul_imm(0, A.mass[i]));
      acc[(size_t)(i - i0) * b + j - j0] = v;
    }
  for (int k = 0; k < A.d0; ++k) {
    std::vector<int> rows, cols;
    for (int i = i0; i < i1; ++i)
      if (A.at(i, k) >= 0) rows.push_back(i);
    for (int j = j0; j < j1; ++j)
      if (A.at(k, j) >= 0) cols.push_back(j);
    if (rows.empty() || cols.empty()) continue;
    for (int i : rows) nl[i - i0] = x.neg(x.load(A.at(i, k)));
    for (int j : cols) {
      const int u = x.load(A.at(k, j));
      for (int i : rows) {
        if (A.at(i, j) < 0) throw std::logic_error("fill pattern not closed");
        int& r = acc[(size_t)(i - i0) * b + j - j0];
        r = x.fma(nl[i - i0], u, r);
        ++x.fmas;
      }
    }
  }
  for (int i = i0; i < i1; ++i)
    for (int j = j0; j < j1; ++j) x.store(gl.dense_item(i, j), acc[(size_t)(i - i0) * b + j - j0]);
}

// The square's columns [j0, j1) of a leading row: assembly and every pivot's
// updates, with the multipliers the row's own task has made.
void emit_row_columns(Ptx& x, const Matrix& A, int i, int j0, int j1) {
  std::vector<int> acc(j1 - j0, -1);
  for (int j = j0; j < j1; ++j) {
    if (A.at(i, j) < 0) continue;
    const int64_t from = A.start[(size_t)i * A.n + j];
    acc[j - j0] = from >= 0 ? x.load(from) : x.constant(0.0);
  }
  for (int k = 0; k < i; ++k) {
    if (A.at(i, k) < 0) continue;
    int nl = -1;
    for (int j = j0; j < j1; ++j) {
      if (A.at(k, j) < 0) continue;
      if (acc[j - j0] < 0) throw std::logic_error("fill pattern not closed");
      if (nl < 0) nl = x.neg(x.load(A.at(i, k)));
      acc[j - j0] = x.fma(nl, x.load(A.at(k, j)), acc[j - j0]);
      ++x.fmas;
    }
  }
  for (int j = j0; j < j1; ++j)
    if (acc[j - j0] >= 0) x.store(A.at(i, j), acc[j - j0]);
}

// The factorization up to the dense square's own elimination. A leading row's
// columns before the square are one task, which alone makes its multipliers
// and pivot; its columns in the square are tasks of about kRowWidth columns
// each, which only the same columns of later rows wait for. With a row as one
// task, the chain of the last leading rows (7,500 multiply-adds of the 210/500
// mechanism) was a quarter of the factorization on a team of sixteen.
std::vector<Task> factor_tasks(const Matrix& A, const GenLayout& gl, int tile) {
  constexpr int kRowWidth = 24;   // columns of a single row at a time
  const int chunk = tile * std::max(1, kRowWidth / tile);
  const int chunks = (A.n - A.d0 + chunk - 1) / chunk;
  std::vector<Task> tasks;
  std::vector<int> row_task(A.n, -1);
  std::vector<int> column_task((size_t)A.n * std::max(1, chunks), -1);
  auto pivots = [&](const std::vector<int>& rows) {
    std::vector<int> ks;
    for (int k = 0; k < std::min(A.d0, rows[0]); ++k)
      for (int i : rows)
        if (A.at(i, k) >= 0) {
          ks.push_back(k);
          break;
        }
    return ks;
  };
  // the tasks that finish the pivots' rows before the square, or in a chunk
  auto before = [&](const std::vector<int>& ks, int c) {
    std::vector<int> after;
    for (int k : ks) {
      const int id = c < 0 ? row_task[k] : column_task[(size_t)k * chunks + c];
      if (id >= 0) after.push_back(id);
    }
    return after;
  };
  for (int i = 0; i < A.d0; ++i) {
    if (A.unit[i]) continue;
    const std::vector<int> rows{i}, ks = pivots(rows);
    row_task[i] = (int)tasks.size();
    tasks.push_back({before(ks, -1), [&A, rows](Ptx& x) { emit_rows(x, A, rows, A.d0, kRowWidth); }});
    for (int c = 0; c < chunks; ++c) {
      const int j0 = A.d0 + c * chunk, j1 = std::min(A.n, j0 + chunk);
      bool any = false;
      for (int j = j0; j < j1 && !any; ++j) any = A.at(i, j) >= 0;
      if (!any) continue;
      std::vector<int> after = before(ks, c);
      if (!ks.empty()) after.push_back(row_task[i]);
      column_task[(size_t)i * chunks + c] = (int)tasks.size();
      tasks.push_back({after, [&A, i, j0, j1](Ptx& x) { emit_row_columns(x, A, i, j0, j1); }});
    }
  }
  for (int i0 = A.d0; i0 < A.n; i0 += tile) {
    const int i1 = std::min(A.n, i0 + tile);
    std::vector<int> rows;
    for (int i = i0; i < i1; ++i) rows.push_back(i);
    const std::vector<int> ks = pivots(rows);
    int mine = -1;
    if (!ks.empty()) {
      mine = (int)tasks.size();
      tasks.push_back({before(ks, -1), [&A, rows, tile](Ptx& x) { emit_rows(x, A, rows, A.d0, tile); }});
    }
    for (int j0 = A.d0; j0 < A.n; j0 += tile) {
      const int j1 = std::min(A.n, j0 + tile);
      std::vector<int> after = before(ks, (j0 - A.d0) / chunk);
      if (mine >= 0) after.push_back(mine);
      tasks.push_back({after, [&A, &gl, i0, i1, j0, j1](Ptx& x) { emit_tile(x, A, gl, i0, i1, j0, j1); }});
    }
  }
  return tasks;
}

// The leading rows' part of a triangular solve in place on the solve vector
// (item xs): row r's value is x_r minus the sum of entry(r, k) x_k over the
// rows k finished before it, in that order, times the item scale(r) where that
// is not -1. Rows finish in ascending order (`up`; the square's rows then lose
// their terms in the leading columns, `block` rows a task) or in descending
// order after the square's rows.
std::vector<Task> triangle_tasks(const Matrix& A, const ScratchLayout& sl, int block, bool up,
                                 std::function<int64_t(int, int)> entry, std::function<int64_t(int)> scale) {
  const int n = A.n, d0 = A.d0;
  std::vector<Task> tasks;
  std::vector<int> maker(n, -1);       // the task that finishes each row (none: before the phase, or never changed)
  // rows [i0, i1) of the vector minus their terms in columns [k0, k1), then,
  // when `finish`, times their scale
  auto emit = [&sl, up, entry, scale](Ptx& x, int i0, int i1, int k0, int k1, bool finish) {
    std::vector<int> acc(i1 - i0, -1);
    for (int m = 0; m < k1 - k0; ++m) {
      const int k = up ? k0 + m : k1 - 1 - m;
      int xk = -1;
      for (int i = i0; i < i1; ++i) {
        const int64_t q = entry(i, k);
        if (q < 0) continue;
        if (xk < 0) xk = x.load(sl.xs + k);
        if (acc[i - i0] < 0) acc[i - i0] = x.load(sl.xs + i);
        acc[i - i0] = x.fma(x.neg(x.load(q)), xk, acc[i - i0]);
      }
    }
    for (int i = i0; i < i1; ++i) {
      if (finish && scale(i) >= 0) {
        if (acc[i - i0] < 0) acc[i - i0] = x.load(sl.xs + i);
        acc[i - i0] = x.mul(acc[i - i0], x.load(scale(i)));
      }
      if (acc[i - i0] >= 0) x.store(sl.xs + i, acc[i - i0]);
    }
  };
  auto terms = [&](int i0, int i1, int k0, int k1) {
    std::vector<int> after;
    bool any = false;
    for (int k = k0; k < k1; ++k)
      for (int i = i0; i < i1; ++i)
        if (entry(i, k) >= 0) {
          any = true;
          if (maker[k] >= 0) after.push_back(maker[k]);
          break;
        }
    return std::make_pair(any, after);
  };
  for (int m = 0; m < d0; ++m) {
    const int i = up ? m : d0 - 1 - m;
    // descending, the terms of the square's rows come first and need no
    // other leading row: a task of their own, all of them in the first step
    int square = -1;
    if (!up && terms(i, i + 1, d0, n).first && terms(i, i + 1, i + 1, d0).first) {
      square = (int)tasks.size();
      tasks.push_back({{}, [=](Ptx& x) { emit(x, i, i + 1, d0, n, false); }});
    }
    const int k0 = up ? 0 : i + 1, k1 = up ? i : square >= 0 ? d0 : n;
    auto [any, after] = terms(i, i + 1, k0, k1);
    if (!any && scale(i) < 0) continue;
    if (square >= 0) after.push_back(square);
    maker[i] = (int)tasks.size();
    tasks.push_back({after, [=](Ptx& x) { emit(x, i, i + 1, k0, k1, true); }});
  }
  for (int i0 = d0; i0 < n && up; i0 += block) {
    const int i1 = std::min(n, i0 + block);
    auto [any, after] = terms(i0, i1, 0, d0);
    if (any) tasks.push_back({after, [=](Ptx& x) { emit(x, i0, i1, 0, d0, false); }});
  }
  return tasks;
}

// The leading parts of (LU)^-1 (L by ascending rows; U by descending rows and
// 1 / pivot) and of (LU)^-T (U^T by ascending rows and 1 / pivot; L^T by
// descending rows), the square's between them being the kernels' loop.
Phase lead_phase(const Matrix& A, const ScratchLayout& sl, int block, bool up, bool transposed) {
  auto entry = [&A, up, transposed](int i, int k) {
    return (up ? k < i : k > i) ? (transposed ? A.at(k, i) : A.at(i, k)) : (int64_t)-1;
  };
  auto scale = [&A, up, transposed](int i) { return up != transposed || A.unit[i] ? (int64_t)-1 : A.at(i, i); };
  return schedule(triangle_tasks(A, sl, block, up, entry, scale));
}

// Items [0, count) in kSegments contiguous ranges, `per` items of a range at
// a time: a batch's loads come before its arithmetic and stores, so that one
// latency covers the batch.
std::vector<std::vector<Emit>> ranges(int count, int per, const std::function<void(Ptx&, int, int)>& batch) {
  std::vector<std::vector<Emit>> out;
  for (int g = 0; g < kSegments; ++g) {
    const int i0 = (int)((int64_t)count * g / kSegments), i1 = (int)((int64_t)count * (g + 1) / kSegments);
    std::vector<Emit> seg;
    for (int i = i0; i < i1; i += per) seg.push_back([=](Ptx& x) { batch(x, i, std::min(i1, i + per)); });
    out.push_back(std::move(seg));
  }
  while (!out.empty() && out.back().empty()) out.pop_back();
  return out;
}

// Rates and forcing at the evaluation point (item yr): r_j = k_j * prod x,
// then F_i = sum of S[i, j] r_j in ascending j, into item ft; the operations
// of the table-driven loops in their order (a leading 0 or 1 and products
// with +-1 are folded, which changes no value). The table-driven loops were
// bound by one dependent chain of loads per row and entry (TS1's attempts
// spent about 90% of their time there): eight intervals of TS1 on 64 cells
// took 297 ms with them and 142 ms with straight-line code on one warp per
// group; one interval of 65,536 cells of the 210/500 mechanism 140.6 ms and
// 128.3 ms.
Phase rhs_phase(const HostTables& t, const ScratchLayout& sl) {
  Phase p;
  p.push_back(ranges(t.R, 8, [&t, &sl](Ptx& x, int j0, int j1) {
    std::vector<std::vector<int>> v(j1 - j0);
    for (int j = j0; j < j1; ++j) {
      v[j - j0].push_back(x.load(sl.kc + j));
      for (int q = 0; q < t.P; ++q)
        if (t.react[(size_t)j * t.P + q] != t.n) v[j - j0].push_back(x.load(sl.yr + t.react[(size_t)j * t.P + q]));
    }
    for (int j = j0; j < j1; ++j) {
      const std::vector<int>& f = v[j - j0];
      int r = f[0];
      if (f.size() > 1) {
        int prod = f[1];
        for (size_t q = 2; q < f.size(); ++q) prod = x.mul(prod, f[q]);
        r = x.mul(f[0], prod);
      }
      x.store(sl.r + j, r);
    }
  }));
  std::vector<Task> rows;
  for (int i = 0; i < t.n; ++i)
    rows.push_back({{}, [&t, &sl, i](Ptx& x) {
      int acc = -1;
      for (int q = t.s_ptr[i]; q < t.s_ptr[i + 1]; ++q) {
        const int r = x.load(sl.r + t.s_rxn[q]);
        const double c = t.s_val[q];
        if (acc < 0) acc = c == 1.0 ? r : c == -1.0 ? x.neg(r) : x.mul_imm(r, c);
        else acc = c == 1.0 ? x.add(acc, r) : c == -1.0 ? x.sub(acc, r) : x.fma_imm(r, c, acc);
      }
      x.store(sl.ft + i, acc < 0 ? x.constant(0.0) : acc);
    }});
  for (auto& s : schedule(rows)) p.push_back(std::move(s));
  return p;
}

// The negated Jacobian values at the evaluation point, in assembly order:
// d[j, p] = k_j * prod of the other reactants, then the sums of -S[i, j] d
// over each entry's terms.
Phase jac_phase(const HostTables& t, const GenLayout& gl) {
  const ScratchLayout& sl = gl.s;
  Phase p;
  p.push_back(ranges(t.R, 8, [&t, &gl, &sl](Ptx& x, int j0, int j1) {
    struct One {
      int item, k;
      std::vector<int> x;
    };
    std::vector<One> ones;
    for (int j = j0; j < j1; ++j) {
      int k = -1;
      std::vector<int> f(t.P, -1);
      for (int a = 0; a < t.P; ++a) {
        const int item = gl.d_item[(size_t)j * t.P + a];
        if (item < 0) continue;
        One o{item, -1, {}};
        if (k < 0) k = x.load(sl.kc + j);
        o.k = k;
        for (int q = 0; q < t.P; ++q) {
          const int s = t.react[(size_t)j * t.P + q];
          if (q == a || s == t.n) continue;
          if (f[q] < 0) f[q] = x.load(sl.yr + s);
          o.x.push_back(f[q]);
        }
        ones.push_back(std::move(o));
      }
    }
    for (const One& o : ones) {
      int d = o.k;
      for (int f : o.x) d = x.mul(d, f);
      x.store(o.item, d);
    }
  }));
  std::vector<Task> entries;
  for (int e = 0; e + 1 < (int)t.jt_ptr.size(); ++e)
    entries.push_back({{}, [&t, &gl, &sl, e](Ptx& x) {
      int acc = -1;
      for (int q = t.jt_ptr[e]; q < t.jt_ptr[e + 1]; ++q) {
        const int jp = t.jt_idx[q];
        const int d = x.load(gl.d_item[jp] >= 0 ? gl.d_item[jp] : sl.kc + jp / t.P);
        const double c = t.jt_val[q];
        if (acc < 0) acc = c == 1.0 ? d : c == -1.0 ? x.neg(d) : x.mul_imm(d, c);
        else acc = c == 1.0 ? x.add(acc, d) : c == -1.0 ? x.sub(acc, d) : x.add(acc, x.mul_imm(d, c));
      }
      x.store(sl.negj + (int64_t)e, acc < 0 ? x.constant(0.0) : acc);
    }});
  for (auto& s : schedule(entries)) p.push_back(std::move(s));
  return p;
}

// The adjoint's forcing product: g = J(yr)^T v (items v, g of the adjoint's
// scratch), reaction by reaction the weights w_j = (S^T v)_j and the rates,
// then species by species the sums of w_j d[j, q] over the reactant slots
// that hold it, in ascending (j, q): the table-driven scatter's order. A
// gather per species needs no order between the warps of a team: with the
// scatter the adjoint ran one warp per group (4,096 cells of the 210/500
// mechanism, one cold interval recorded and reversed: 1.42 s, now 0.315 s).
Phase vjp_phase(const HostTables& t, const GenLayout& gl, const AdjLayout& al) {
  const ScratchLayout& sl = gl.s;
  Phase p;
  p.push_back(ranges(t.R, 4, [&t, &gl, &sl, &al](Ptx& x, int j0, int j1) {
    for (int j = j0; j < j1; ++j) {
      const int k = x.load(sl.kc + j);
      std::vector<int> f(t.P, -1);
      for (int q = 0; q < t.P; ++q)
        if (t.react[(size_t)j * t.P + q] != t.n) f[q] = x.load(sl.yr + t.react[(size_t)j * t.P + q]);
      int w = -1;
      for (int e = t.st_ptr[j]; e < t.st_ptr[j + 1]; ++e) {
        const int v = x.load(al.v + t.st_sp[e]);
        w = w < 0 ? x.mul_imm(v, t.st_val[e]) : x.fma_imm(v, t.st_val[e], w);
      }
      x.store(al.w + j, w < 0 ? x.constant(0.0) : w);
      int rate = k;
      for (int q = 0; q < t.P; ++q)
        if (f[q] >= 0) rate = x.mul(rate, f[q]);
      x.store(al.rate + j, rate);
      for (int a = 0; a < t.P; ++a) {
        if (gl.d_item[(size_t)j * t.P + a] < 0) continue;
        int d = k;
        for (int q = 0; q < t.P; ++q)
          if (q != a && f[q] >= 0) d = x.mul(d, f[q]);
        x.store(gl.d_item[(size_t)j * t.P + a], d);
      }
    }
  }));
  std::vector<std::vector<int>> uses(t.n);
  for (int jq = 0; jq < t.R * t.P; ++jq)
    if (t.react[jq] != t.n && t.st_ptr[jq / t.P] < t.st_ptr[jq / t.P + 1]) uses[t.react[jq]].push_back(jq);
  std::vector<Task> rows;
  for (int i = 0; i < t.n; ++i)
    rows.push_back({{}, [&t, &gl, &sl, &al, i, u = uses[i]](Ptx& x) {
      int acc = -1;
      for (int jq : u) {
        const int w = x.load(al.w + jq / t.P);
        const int d = x.load(gl.d_item[jq] >= 0 ? gl.d_item[jq] : sl.kc + jq / t.P);
        acc = acc < 0 ? x.mul(w, d) : x.fma(w, d, acc);
      }
      x.store(al.g + i, acc < 0 ? x.constant(0.0) : acc);
    }});
  for (auto& s : schedule(rows)) p.push_back(std::move(s));
  return p;
}

// The second derivatives of the Jacobian at yr contracted with jbar: dbar, the
// adjoint of every d[j, q], and the reactions' log k derivatives (item w),
// then ybar gains dbar[j, q] dd over the slots q2 != q that hold each species,
// in ascending (j, q, q2).
Phase hvp_phase(const HostTables& t, const GenLayout& gl, const AdjLayout& al) {
  const ScratchLayout& sl = gl.s;
  // the Jacobian entries each d[j, q] enters, in ascending order
  auto terms = std::make_shared<std::vector<std::vector<std::pair<int, double>>>>((size_t)t.R * t.P);
  for (int e = 0; e + 1 < (int)t.jt_ptr.size(); ++e)
    for (int q = t.jt_ptr[e]; q < t.jt_ptr[e + 1]; ++q) (*terms)[t.jt_idx[q]].push_back({e, -t.jt_val[q]});
  Phase p;
  std::vector<Task> reactions;
  for (int j = 0; j < t.R; ++j)
    reactions.push_back({{}, [&t, &sl, &al, terms, j](Ptx& x) {
      const int k = x.load(sl.kc + j);
      std::vector<int> f(t.P, -1);
      for (int q = 0; q < t.P; ++q)
        if (t.react[(size_t)j * t.P + q] != t.n) f[q] = x.load(sl.yr + t.react[(size_t)j * t.P + q]);
      int th = -1;
      for (int q = 0; q < t.P; ++q) {
        if (f[q] < 0) continue;
        int db = -1;
        for (const auto& [e, c] : (*terms)[(size_t)j * t.P + q]) {
          const int v = x.load(al.jbar + e);
          db = db < 0 ? x.mul_imm(v, c) : x.fma_imm(v, c, db);
        }
        if (db < 0) db = x.constant(0.0);
        x.store(al.dbar + (int64_t)j * t.P + q, db);
        int d = k;
        for (int q2 = 0; q2 < t.P; ++q2)
          if (q2 != q && f[q2] >= 0) d = x.mul(d, f[q2]);
        th = th < 0 ? x.mul(db, d) : x.fma(db, d, th);
      }
      x.store(al.w + j, th < 0 ? x.constant(0.0) : th);
    }});
  for (auto& s : schedule(reactions)) p.push_back(std::move(s));
  struct Use {
    int jq, q2;
  };
  std::vector<std::vector<Use>> uses(t.n);
  for (int j = 0; j < t.R; ++j)
    for (int q = 0; q < t.P; ++q) {
      if (t.react[(size_t)j * t.P + q] == t.n || (*terms)[(size_t)j * t.P + q].empty()) continue;
      for (int q2 = 0; q2 < t.P; ++q2)
        if (q2 != q && t.react[(size_t)j * t.P + q2] != t.n)
          uses[t.react[(size_t)j * t.P + q2]].push_back({j * t.P + q, q2});
    }
  std::vector<Task> rows;
  for (int i = 0; i < t.n; ++i) {
    if (uses[i].empty()) continue;
    rows.push_back({{}, [&t, &sl, &al, i, u = uses[i]](Ptx& x) {
      int acc = x.load(al.ybar + i);
      for (const Use& o : u) {
        const int j = o.jq / t.P;
        const int db = x.load(al.dbar + o.jq);
        int dd = x.load(sl.kc + j);
        for (int q3 = 0; q3 < t.P; ++q3)
          if (q3 != o.jq % t.P && q3 != o.q2 && t.react[(size_t)j * t.P + q3] != t.n)
            dd = x.mul(dd, x.load(sl.yr + t.react[(size_t)j * t.P + q3]));
        acc = x.fma(db, dd, acc);
      }
      x.store(al.ybar + i, acc);
    }});
  }
  for (auto& s : schedule(rows)) p.push_back(std::move(s));
  return p;
}

// One phase of every mechanism as a function that all warps of a team call:
//   .visible .func name(base, [alpha,] warp, warps, mech)
// A team barrier, then mechanism mech's steps: warp w runs the segments w,
// w + warps, ... of a step, and a team barrier ends it. Runs of tasks of
// piece_lines instructions are functions of their own: ptxas optimizes those
// side by side, and does not hoist one tile's loads over another's arithmetic
// (segments compiled whole spilled up to 5 KB).
std::string phase_function(const std::string& name, bool alpha, const std::vector<Phase>& mechs, size_t piece_lines,
                           int64_t* fmas) {
  std::string pieces, body;
  Ptx x;
  int labels = 0;
  auto label = [&](const char* what, int id) { return "$" + name + "_" + what + std::to_string(id); };
  const std::string regs = ";\n\t.reg .b64 %p;\n\t.reg .b64 %b;\n\t.reg .b64 %a;\n";
  // the block's barrier, or the cluster's for a team of several blocks
  const std::string barrier =
      "\t@%team bar.sync 0;\n\t@%clus barrier.cluster.arrive.release.aligned;\n"
      "\t@%clus barrier.cluster.wait.acquire.aligned;\n";
  for (size_t m = 0; m < mechs.size(); ++m) {
    if (m + 1 < mechs.size())
      body += "\tsetp.ne.s32 %q, %m, " + std::to_string(m) + ";\n\t@%q bra " + label("m", (int)m + 1) + ";\n";
    for (size_t s = 0; s < mechs[m].size(); ++s) {
      const auto& segs = mechs[m][s];
      const int id = labels++, count = (int)segs.size();
      std::string table;
      for (int g = 0; g < count; ++g) table += (g ? ", " : "") + label(("g" + std::to_string(id) + "_").c_str(), g);
      body += "\tmov.u32 %s, %w;\n" + label("l", id) + ":\n\tsetp.ge.u32 %q, %s, " + std::to_string(count) +
              ";\n\t@%q bra " + label("e", id) + ";\n";
      if (count > 1) body += label("t", id) + ": .branchtargets " + table + ";\n\tbrx.idx.uni %s, " + label("t", id) + ";\n";
      for (int g = 0; g < count; ++g) {
        body += label(("g" + std::to_string(id) + "_").c_str(), g) + ":\n";
        // tasks in order, gathered into runs of about piece_lines
        // instructions: a run that reaches that is a function of its own
        for (size_t q = 0, part = 0; q < segs[g].size(); ++part) {
          Ptx own;
          size_t lines = 0, q0 = q;
          while (q < segs[g].size() && lines < piece_lines) {
            segs[g][q++](own);
            lines = (size_t)std::count(own.body.begin(), own.body.end(), '\n');
          }
          *fmas += own.fmas;
          if (lines < piece_lines) {
            for (; q0 < q; ++q0) segs[g][q0](x);
            body += x.body;
            x.body.clear();
            continue;
          }
          const std::string piece =
              name + "_" + std::to_string(id) + "_" + std::to_string(g) + "_" + std::to_string(part);
          pieces += ".func " + piece + "(.param .b64 " + piece + "_base, .param .b64 " + piece + "_alpha)\n{\n" +
                    "\t.reg .f64 %d<" + std::to_string(own.next + 1) + ">" + regs + "\tld.param.b64 %b, [" + piece +
                    "_base];\n\tld.param.b64 %a, [" + piece + "_alpha];\n\tmov.b64 %d0, %a;\n" + own.body +
                    "\tret;\n}\n\n";
          body += "\t{\n\t.param .b64 fo_arg_base;\n\t.param .b64 fo_arg_alpha;\n\tst.param.b64 [fo_arg_base], %b;\n"
                  "\tst.param.b64 [fo_arg_alpha], %a;\n\tcall.uni " + piece + ", (fo_arg_base, fo_arg_alpha);\n\t}\n";
        }
        body += "\tbra " + label("n", id) + ";\n";
      }
      body += label("n", id) + ":\n\tadd.u32 %s, %s, %nw;\n\tbra " + label("l", id) + ";\n" + label("e", id) +
              ":\n" + barrier;
    }
    body += "\tret;\n";
    if (m + 1 < mechs.size()) body += label("m", (int)m + 1) + ":\n";
  }
  auto param = [&](const char* what) { return name + "_" + what; };
  std::string s = pieces + ".visible .func " + name + "(.param .b64 " + param("base") +
                  (alpha ? ", .param .b64 " + param("alpha") : "") + ", .param .b32 " + param("warp") +
                  ", .param .b32 " + param("warps") + ", .param .b32 " + param("mech") + ")\n{\n\t.reg .f64 %d<" +
                  std::to_string(x.next + 1) + ">" + regs +
                  "\t.reg .b32 %m;\n\t.reg .b32 %w;\n\t.reg .b32 %nw;\n\t.reg .b32 %s;\n"
                  "\t.reg .pred %q;\n\t.reg .pred %team;\n\t.reg .pred %clus;\n\tld.param.b64 %p, [" + param("base") + "];\n" +
                  (alpha ? "\tld.param.b64 %a, [" + param("alpha") + "];\n" : "\tmov.b64 %a, 0x3FF0000000000000;\n") +
                  "\tmov.b64 %d0, %a;\n\tld.param.b32 %w, [" + param("warp") + "];\n\tld.param.b32 %nw, [" +
                  param("warps") + "];\n\tld.param.b32 %m, [" + param("mech") +
                  "];\n\tcvta.to.global.u64 %b, %p;\n\tsetp.gt.u32 %clus, %nw, " + std::to_string(kBlockWarps) +
                  ";\n\tsetp.gt.u32 %team, %nw, 1;\n\t@%clus setp.ne.u32 %team, %nw, %nw;\n" + barrier;
  return s + body + "}\n\n";
}

}  // namespace

std::string generate_ptx(const std::vector<const HostTables*>& ts, const std::vector<GenOptions>& os,
                         int64_t* fma_count) {
  if (ts.empty() || os.size() != ts.size()) throw std::invalid_argument("one set of options per mechanism");
  for (const GenOptions& o : os)
    if (o.tile < 1 || o.tile > 16 || o.solve_block < 1 || o.solve_block > 64 || o.piece_lines < 1)
      throw std::invalid_argument("generation options out of range");
  const size_t count = ts.size();
  std::vector<GenLayout> layouts;
  std::vector<AdjLayout> adjoints;
  std::vector<Matrix> full, proj;
  for (const HostTables* t : ts) {
    layouts.push_back(gen_layout_of(*t));
    adjoints.push_back(adjoint_layout(*t, 0));
  }
  for (size_t m = 0; m < count; ++m) {
    full.push_back(full_matrix(*ts[m], layouts[m]));
    proj.push_back(projection_matrix(*ts[m], layouts[m]));
  }
  std::vector<Phase> rhs, jac, factor, pfactor, vjp, hvp;
  // leading parts of the solves: [full or projection][transposed][up or down]
  std::vector<Phase> lead[2][2][2];
  int64_t expected = 0;
  for (size_t m = 0; m < count; ++m) {
    const HostTables& t = *ts[m];
    const GenLayout& gl = layouts[m];
    const GenOptions& o = os[m];
    rhs.push_back(rhs_phase(t, gl.s));
    jac.push_back(jac_phase(t, gl));
    vjp.push_back(vjp_phase(t, gl, adjoints[m]));
    hvp.push_back(hvp_phase(t, gl, adjoints[m]));
    factor.push_back(schedule(factor_tasks(full[m], gl, o.tile)));
    bool constrained = false;
    for (double v : t.mass) constrained = constrained || v == 0.0;
    pfactor.push_back(constrained ? schedule(factor_tasks(proj[m], gl, o.tile)) : Phase());
    for (int p = 0; p < 2; ++p)
      for (int tr = 0; tr < 2; ++tr)
        for (int down = 0; down < 2; ++down)
          lead[p][tr][down].push_back(p && !constrained ? Phase()
                                                        : lead_phase(p ? proj[m] : full[m], gl.s, o.solve_block, !down, tr != 0));
    // the multiply-adds of the pivots before the dense square
    for (int i = 0; i < t.n; ++i)
      for (int q = t.lu_row_ptr[i]; q < t.lu_diag[i]; ++q)
        if (t.lu_col[q] < gl.d0) expected += t.lu_row_ptr[t.lu_col[q] + 1] - t.lu_diag[t.lu_col[q]] - 1;
  }
  size_t lines = 0;
  for (const GenOptions& o : os) lines = std::max(lines, (size_t)o.piece_lines);
  std::string out = ".version 9.0\n.target sm_103a\n.address_size 64\n\n";
  int64_t nfma = 0, ignored = 0;
  out += phase_function("fo_gen_factor", true, factor, lines, &nfma);
  if (nfma != expected) throw std::logic_error("generated factorization does not match the symbolic count");
  if (fma_count) {
    *fma_count = 0;
    for (const HostTables* t : ts) *fma_count += t->lu_fma;
  }
  for (int p = 0; p < 2; ++p)
    for (int tr = 0; tr < 2; ++tr)
      for (int down = 0; down < 2; ++down)
        out += phase_function(std::string("fo_gen_solve") + (tr ? "_t" : "") + (p ? "_p" : "") + (down ? "_down" : "_up"),
                              false, lead[p][tr][down], lines, &ignored);
  out += phase_function("fo_gen_rhs", false, rhs, lines, &ignored);
  out += phase_function("fo_gen_jac", false, jac, lines, &ignored);
  out += phase_function("fo_gen_vjp", false, vjp, lines, &ignored);
  out += phase_function("fo_gen_hvp", false, hvp, lines, &ignored);
  out += phase_function("fo_gen_factor_p", false, pfactor, lines, &ignored);
  return out;
}

std::string generate_ptx(const HostTables& t, const GenOptions& o, int64_t* fma_count) {
  return generate_ptx(std::vector<const HostTables*>{&t}, std::vector<GenOptions>{o}, fma_count);
}

}  // namespace fo
