// The per-lane scratch layout of a plan, shared by the launch code (abi.cu)
// and the code generator (codegen.cpp), which bakes its offsets into the
// generated functions.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "device.cuh"
#include "symbolic.h"

namespace fo {

inline ScratchLayout layout_of(const HostTables& t) {
  ScratchLayout s;
  int64_t o = 0;
  s.lu = o; o += (int64_t)t.lu_col.size();
  s.negj = o; o += (int64_t)t.j_col.size();
  s.d = o; o += (int64_t)t.R * t.P;
  s.r = o; o += t.R;
  s.y = o; o += t.n;
  s.ynew = o; o += t.n;
  s.f0 = o; o += t.n;
  s.ft = o; o += t.n;
  s.yr = o; o += t.n;
  s.k = o; o += 4LL * t.n;
  s.xs = o; o += t.n;
  s.kc = 0;
  s.items = o;
  return s;
}

// The layout of the generated variant, in no more items than layout_of (one
// workspace serves both). The generated evaluations keep the interval's rate
// constants (kc), so that every operand of theirs is at an immediate offset
// from the slot's base, and store only the partial derivatives that are
// products (a unimolecular reaction's is its rate constant); those and the
// rates are never live together and share their items.
struct GenLayout {
  ScratchLayout s;
  std::vector<int32_t> d_item;  // R*P: item of d[j, p], or -1 where it is k_j itself or not used
};

inline GenLayout gen_layout_of(const HostTables& t) {
  GenLayout g;
  g.s = layout_of(t);
  g.d_item.assign((size_t)t.R * t.P, -1);
  int64_t nd = 0;
  std::vector<char> used((size_t)t.R * t.P, 0);
  for (int32_t q : t.jt_idx) used[q] = 1;
  for (int j = 0; j < t.R; ++j) {
    int factors = 0;
    for (int q = 0; q < t.P; ++q) factors += t.react[(size_t)j * t.P + q] != t.n ? 1 : 0;
    for (int a = 0; a < t.P; ++a) {
      const int others = factors - (t.react[(size_t)j * t.P + a] != t.n ? 1 : 0);
      if (used[(size_t)j * t.P + a] && others > 0) g.d_item[(size_t)j * t.P + a] = (int32_t)(g.s.d + nd++);
    }
  }
  g.s.r = g.s.d;
  g.s.kc = g.s.d + std::max<int64_t>(nd, t.R);
  return g;
}

}  // namespace fo
