// The generated variant's scratch layout, and the size of the dense square.
#include "layout.h"

#include <algorithm>
#include <stdexcept>

namespace fo {
namespace {

// Entries and multiply-adds of the LU around a trailing square that starts
// at row d0.
struct Split {
  int64_t outside = 0;  // entries outside the square
  int64_t fma = 0;      // multiply-adds of the pivots before it
  int64_t lead = 0;     // those of the rows before it
};

Split split_at(const HostTables& t, int d0) {
  Split s;
  for (int i = 0; i < t.n; ++i)
    for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q) {
      const int k = t.lu_col[q];
      if (i < d0 || k < d0) ++s.outside;
      if (q >= t.lu_diag[i] || k >= d0) continue;
      const int64_t c = t.lu_row_ptr[k + 1] - t.lu_diag[k] - 1;
      s.fma += c;
      if (i < d0) s.lead += c;
    }
  return s;
}

// Blocks of the dense square. The square is eliminated by a loop that treats
// it as full, the rows before it by straight-line code in dependency order.
// A larger square multiplies more zeros, a smaller one leaves more work to
// the rows before it, which have little parallelism between them; the size
// taken minimizes the multiply-adds done plus those of the leading rows. For
// the 210/500 mechanism: 72 rows, 210 k (60 rows: 224 k, 84 rows: 241 k).
int dense_blocks(const HostTables& t, int64_t slack) {
  int best = 0;
  int64_t best_cost = -1;
  for (int nb = 0; nb * kDenseBlock <= t.n; ++nb) {
    const int64_t D = (int64_t)nb * kDenseBlock;
    const Split s = split_at(t, (int)(t.n - D));
    if (s.outside + D * D > (int64_t)t.lu_col.size() + slack) continue;
    const int64_t cost = s.fma + s.lead + D * (D - 1) * (2 * D - 1) / 6;
    if (best_cost < 0 || cost < best_cost) {
      best = nb;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace

int64_t GenLayout::dense_item(int i, int j) const {
  const int r = i - d0, c = j - d0;
  return s.dn + (int64_t)(r / kDenseBlock * s.nb + c / kDenseBlock) * kDenseBlock * kDenseBlock +
         r % kDenseBlock * kDenseBlock + c % kDenseBlock;
}

GenLayout gen_layout_of(const HostTables& t) {
  const ScratchLayout table = layout_of(t);
  GenLayout g;
  // the partial derivatives that are products
  std::vector<char> used((size_t)t.R * t.P, 0);
  for (int32_t q : t.jt_idx) used[q] = 1;
  for (int j = 0; j < t.R; ++j)
    if (t.st_ptr[j] < t.st_ptr[j + 1])
      for (int a = 0; a < t.P; ++a) used[(size_t)j * t.P + a] = t.react[(size_t)j * t.P + a] != t.n;
  std::vector<int64_t> product((size_t)t.R * t.P, -1);
  int64_t nd = 0;
  for (int j = 0; j < t.R; ++j) {
    int factors = 0;
    for (int q = 0; q < t.P; ++q) factors += t.react[(size_t)j * t.P + q] != t.n ? 1 : 0;
    for (int a = 0; a < t.P; ++a) {
      const size_t jp = (size_t)j * t.P + a;
      const int others = factors - (t.react[jp] != t.n ? 1 : 0);
      if (used[jp] && others > 0) product[jp] = nd++;
    }
  }
  const int64_t shared = std::max<int64_t>(nd, t.R);  // the products and the rates
  ScratchLayout& s = g.s;
  s.nb = dense_blocks(t, (int64_t)t.R * t.P - shared);
  g.d0 = t.n - s.nb * kDenseBlock;
  int64_t o = 0;
  s.lu = o;
  g.lu_item.assign(t.lu_col.size(), -1);
  for (int i = 0; i < t.n; ++i)
    for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q)
      if (i < g.d0 || t.lu_col[q] < g.d0) g.lu_item[q] = o++;
  s.dn = o;
  for (int i = g.d0; i < t.n; ++i)
    for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q)
      if (t.lu_col[q] >= g.d0) g.lu_item[q] = g.dense_item(i, t.lu_col[q]);
  o += (int64_t)s.nb * s.nb * kDenseBlock * kDenseBlock;
  s.negj = o; o += (int64_t)t.j_col.size();
  s.d = s.r = o; o += shared;
  s.kc = o; o += t.R;
  s.y = o; o += t.n;
  s.ynew = o; o += t.n;
  s.f0 = o; o += t.n;
  s.ft = o; o += t.n;
  s.yr = o; o += t.n;
  s.k = o; o += 4LL * t.n;
  s.xs = o; o += t.n;
  if (o > table.items) throw std::logic_error("the generated layout exceeds the plan's scratch");
  s.items = table.items;
  g.d_item.assign((size_t)t.R * t.P, -1);
  for (size_t q = 0; q < product.size(); ++q)
    if (product[q] >= 0) g.d_item[q] = (int32_t)(s.d + product[q]);
  return g;
}

AdjLayout adjoint_layout(const HostTables& t, int max_steps) {
  AdjLayout a;
  bool constrained = false;
  for (double m : t.mass) constrained = constrained || m == 0.0;
  int64_t o = layout_of(t).items;
  a.u = o; o += 4LL * t.n;
  a.kbar = o; o += 4LL * t.n;
  a.fbar = o; o += 4LL * t.n;
  a.ybar = o; o += t.n;
  a.g = o; o += t.n;
  a.v = o; o += t.n;
  a.jbar = o; o += (int64_t)t.j_col.size();
  a.dbar = o; o += (int64_t)t.R * t.P;
  a.w = o; o += t.R;
  a.rate = o; o += t.R;
  a.pdelta = o; o += constrained ? t.n : 0;
  a.pmu = o; o += constrained ? t.n : 0;
  a.yp = o; o += constrained ? (int64_t)kMaxProjectionUpdates * t.n : 0;
  a.ys = o; o += (int64_t)max_steps * t.n;
  a.items = o;
  return a;
}

}  // namespace fo
