// Per-mechanism code generation: the evaluations, the factorization of
// alpha*M - J and the triangular solves of one mechanism as straight-line PTX,
// every operand at an immediate offset from a lane's base pointer. The integrator kernel compiled
// as relocatable device code (generated.cu) calls them; jit.cpp links the
// two into one module per mechanism.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "symbolic.h"

namespace fo {

// Segments of a step of generated work: the most warps of a team that a step
// can use (half of those of a cluster of eight blocks).
constexpr int kSegments = 64;

// Warps of a block; a larger team is a cluster of blocks of this many.
constexpr int kBlockWarps = 16;

struct GenOptions {
  // rows and columns of the register tiles of the factorization
  int tile = 6;
  // rows of a block of the triangular solves
  int solve_block = 4;
  // instructions of consecutive tasks compiled as a function of their own
  int piece_lines = 400;
};

// PTX (ISA 9.0, sm_103a) of the phases of one mechanism, each a function that
// every warp of a group's team calls with its index and the team's size:
//   .visible .func name(.param .b64 base, .param .b32 warp, .param .b32 warps, .param .b32 mech)
// base points at this lane's item 0 of its scratch slot, laid out item-major
// with 32 lanes (item q at byte offset 256 q) by GenLayout (layout.h). Every
// phase begins and ends with the team's barrier (none for a team of one, the
// cluster's for a team of more than kBlockWarps).
//   fo_gen_rhs       forcing at the point in item yr, into item ft
//   fo_gen_jac       negated Jacobian values at yr, into item negj
//   fo_gen_factor    (base, alpha, ...) assembles alpha*M - J and factors it up
//                    to the dense square, which it leaves assembled and updated
//                    (dense_lu finishes it)
//   fo_gen_solve_up, fo_gen_solve_down
//                    the leading rows' part of (LU)^-1 on the solve vector (item
//                    xs): before and after the square's (square_triangle)
//   fo_gen_solve_t_up, fo_gen_solve_t_down
//                    the same of (LU)^-T, for the adjoint
//   fo_gen_vjp       the adjoint's J(yr)^T v, weights and rates
//   fo_gen_hvp       the adjoint's second derivatives of the Jacobian at yr
//   fo_gen_factor_p, fo_gen_solve_p_up, ..., fo_gen_solve_t_p_down
//                    the same for the projection's algebraic-rows-only matrix,
//                    which has no square (empty for unconstrained mechanisms)
// `mech` is ignored (one mechanism).
std::string generate_ptx(const HostTables& t, const GenOptions& o, int64_t* fma_count = nullptr);

// The same for several mechanisms in one module: `mech` is the mechanism's
// index in `ts` and selects its code.
std::string generate_ptx(const std::vector<const HostTables*>& ts, const std::vector<GenOptions>& os,
                         int64_t* fma_count = nullptr);

}  // namespace fo
