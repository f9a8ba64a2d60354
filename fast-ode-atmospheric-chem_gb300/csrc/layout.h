// The per-lane scratch layouts of a plan, shared by the launch code (abi.cu)
// and the code generator (codegen.cpp), which bakes its offsets into the
// generated functions.
#pragma once

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
  s.dn = 0;
  s.nb = 0;
  s.items = o;
  return s;
}

// The layout of the generated variant, in no more items than layout_of (one
// workspace serves both). The generated evaluations keep the interval's rate
// constants (kc), so that every operand of theirs is at an immediate offset
// from the slot's base, and store only the partial derivatives that are
// products (a unimolecular reaction's is its rate constant); those and the
// rates are never live together and share their items. The trailing
// kDenseBlock * nb rows and columns of the LU are stored as a dense square of
// nb x nb blocks (item dn), block (bi, bj) as kDenseBlock^2 items, row-major,
// at (bi * nb + bj) * kDenseBlock^2; the other entries keep their order.
struct GenLayout {
  ScratchLayout s;
  int d0 = 0;                    // first row of the dense square (n: none)
  std::vector<int32_t> d_item;   // R*P: item of d[j, p], or -1 where it is k_j itself or not used
  std::vector<int64_t> lu_item;  // item of each LU entry
  // item of (i, j) of the dense square (structural zeros included)
  int64_t dense_item(int i, int j) const;
};

GenLayout gen_layout_of(const HostTables& t);

AdjLayout adjoint_layout(const HostTables& t, int max_steps);

}  // namespace fo
