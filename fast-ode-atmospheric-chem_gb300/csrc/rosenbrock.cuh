// Device functions of the Rosenbrock integrator: the mechanism evaluations,
// the sparse LU and its solves, the stage loop, the error norm, the
// controller and the projection of one group over one interval
// (fastode/solvers.py:37-415, chem.py:86-102, linalg.py:15-81), shared by the
// forward kernels (integrator.cu) and the adjoint kernels (adjoint.cu).
// Each translation unit that includes this file gets its own copy.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include <cmath>
#include <cstdint>

#include "device.cuh"
#include "fastode_gb300.h"
#include "tableaus.h"

#ifdef FO_LINK_GENERATED
// The mechanism's generated phases (codegen.h), linked in per mechanism:
// `base` is this lane's item 0 of its scratch slot (32 lanes), `warp` of
// `warps` the caller's place in the group's team, `mech` the mechanism's
// index in the module (several mechanisms share one).
extern "C" {
__device__ void fo_gen_rhs(double* base, int warp, int warps, int mech);
__device__ void fo_gen_jac(double* base, int warp, int warps, int mech);
__device__ void fo_gen_factor(double* base, double alpha, int warp, int warps, int mech);
__device__ void fo_gen_solve_up(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_down(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_t_up(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_t_down(double* base, int warp, int warps, int mech);
__device__ void fo_gen_factor_p(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_p_up(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_p_down(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_t_p_up(double* base, int warp, int warps, int mech);
__device__ void fo_gen_solve_t_p_down(double* base, int warp, int warps, int mech);
__device__ void fo_gen_vjp(double* base, int warp, int warps, int mech);
__device__ void fo_gen_hvp(double* base, int warp, int warps, int mech);
}
// The team: the warps of the block (blockDim = 32 x warps), or of a cluster of
// such blocks, all holding the group's cells. Loops over species give warp w
// the species i = w mod warps (a power of two), so that elementwise loops hand
// no value to another warp.
__device__ __forceinline__ int cluster_rank() {
  int r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ int cluster_blocks() {
  int r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
#define TEAM_W ((int)threadIdx.y + cluster_rank() * (int)blockDim.y)
#define TEAM_N ((int)blockDim.y * cluster_blocks())
// the block's own warps (what each block of a cluster computes for itself)
#define BLOCK_W ((int)threadIdx.y)
#define BLOCK_N ((int)blockDim.y)
#else
#define TEAM_W 0
#define TEAM_N 1
#define BLOCK_W 0
#define BLOCK_N 1
#endif

namespace fo {
// internal linkage: every translation unit that includes this file keeps its
// own copy of these device functions
namespace {


#define SCR(base, item) (base)[(int64_t)(item) * L + lane]
#define WROW(c) w[(c) * L + lane]

__device__ __forceinline__ double pymin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double pymax(double a, double b) { return (b > a) ? b : a; }
// numpy.maximum: NaN if either operand is NaN
__device__ __forceinline__ double npmax(double a, double b) {
  if (a != a) return a;
  if (b != b) return b;
  return (a > b) ? a : b;
}
// numpy.maximum(y, 0.0): keeps NaN, maps -0.0 to 0.0
__device__ __forceinline__ double clamp0(double y) { return (y <= 0.0) ? 0.0 : y; }

// fastode/solvers.py:46-51
__device__ __forceinline__ double quantize_step(double h, double interval) {
  if (h >= interval) return interval;
  double q = ceil(__dsub_rn(__ddiv_rn(interval, h), 1.0e-9));
  if (!(q >= 1.0)) q = 1.0;
  return __ddiv_rn(interval, q);
}

// The team's barrier, and its one thread that writes a group's results.
__device__ __forceinline__ void team_sync() {
#ifdef FO_LINK_GENERATED
  if (cluster_blocks() > 1) {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::
            : "memory");
    return;
  }
#endif
  if (TEAM_N > 1) __syncthreads();
}
__device__ __forceinline__ bool cluster_team() {
#ifdef FO_LINK_GENERATED
  return cluster_blocks() > 1;
#else
  return false;
#endif
}
__device__ __forceinline__ bool team_leader() { return threadIdx.x == 0 && TEAM_W == 0; }

struct Lane {
  int lane;      // thread index in the block
  int L;         // lanes per block
  int64_t cell;  // global cell index (clamped into the group for idle lanes)
  bool active;   // this lane owns a real cell of the group
};

// Rates r_j = k_j * prod(x[react[j, :]]) (fastode/chem.py:86-87). The
// arrays are distinct scratch items, so the loads of several reactions can be
// in flight together.
__device__ void eval_rates(const SolveParams& p, const Lane& ln, const double* __restrict__ x,
                           double* __restrict__ r) {
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n, R = p.t.R, P = p.t.P;
  const double* __restrict__ kc = p.k + ln.cell * p.kcs;
#pragma unroll 4
  for (int j = 0; j < R; ++j) {
    double prod = 1.0;
    for (int q = 0; q < P; ++q) {
      int s = __ldg(p.t.react + j * P + q);
      if (s != n) prod = __dmul_rn(prod, SCR(x, s));
    }
    SCR(r, j) = __dmul_rn(__ldg(kc + (int64_t)j * p.krs), prod);
  }
}

// Forcing F = S r, species rows of the permuted stoichiometry
// (fastode/chem.py:89-90). Each row's rates are loaded eight at a time
// before they are summed in order, so their latencies overlap.
__device__ void eval_forcing(const SolveParams& p, const Lane& ln, const double* __restrict__ r,
                             double* __restrict__ f) {
  constexpr int kBatch = 8;
  const int L = ln.L, lane = ln.lane;
  for (int i = 0; i < p.t.n; ++i) {
    double acc = 0.0;
    const int q1 = __ldg(p.t.s_ptr + i + 1);
    int q = __ldg(p.t.s_ptr + i);
    for (; q + kBatch <= q1; q += kBatch) {
      double v[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) v[b] = SCR(r, __ldg(p.t.s_rxn + q + b));
#pragma unroll
      for (int b = 0; b < kBatch; ++b) acc = fma(__ldg(p.t.s_val + q + b), v[b], acc);
    }
    for (; q < q1; ++q) acc = fma(__ldg(p.t.s_val + q), SCR(r, __ldg(p.t.s_rxn + q)), acc);
    SCR(f, i) = acc;
  }
}

// v = u for a per-lane vector of n items, kBatch loads in flight.
__device__ __forceinline__ void copy_items(const Lane& ln, int n, const double* u, double* v) {
  constexpr int kBatch = 8;
  const int L = ln.L, lane = ln.lane;
  for (int i = TEAM_W; i < n; i += kBatch * TEAM_N) {
    double b[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (i + q * TEAM_N < n) b[q] = SCR(u, i + q * TEAM_N);
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (i + q * TEAM_N < n) SCR(v, i + q * TEAM_N) = b[q];
  }
}

// What the generated evaluations keep for a group's interval: its rate
// constants in the slot (item kc).
__device__ __forceinline__ void load_rate_constants(const SolveParams& p, const Lane& ln, double* scr) {
#ifdef FO_LINK_GENERATED
  constexpr int kBatch = 8;
  const int L = ln.L, lane = ln.lane;
  const double* __restrict__ kc = p.k + ln.cell * p.kcs;
  double* out = scr + p.sl.kc * L;
  for (int j = TEAM_W; j < p.t.R; j += kBatch * TEAM_N) {
    double b[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (j + q * TEAM_N < p.t.R) b[q] = __ldg(kc + (int64_t)(j + q * TEAM_N) * p.krs);
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (j + q * TEAM_N < p.t.R) SCR(out, j + q * TEAM_N) = b[q];
  }
#endif
}

// F(x) into f. The generated form evaluates at the slot's point yr (x is
// copied there) and leaves the point for eval_negjac, which follows at the
// same x wherever it is called.
__device__ __noinline__ void eval_rhs(const SolveParams& p, const Lane& ln, const double* x, double* r, double* f) {
#ifdef FO_LINK_GENERATED
  double* base = r - p.sl.r * ln.L;
  double* yr = base + p.sl.yr * ln.L;
  double* ft = base + p.sl.ft * ln.L;
  if (x != yr) copy_items(ln, p.t.n, x, yr);
  fo_gen_rhs(base + ln.lane, TEAM_W, TEAM_N, p.o.gen_index);
  if (f != ft) copy_items(ln, p.t.n, ft, f);
#else
  eval_rates(p, ln, x, r);
  eval_forcing(p, ln, r, f);
#endif
}

// Negated Jacobian values in assembly order: d[j,p] = k_j prod_{q != p} x_q,
// then -J = sum of (-S[i,j]) d[j,p] over the map's terms
// (fastode/chem.py:92-102).
__device__ __noinline__ void eval_negjac(const SolveParams& p, const Lane& ln, const double* __restrict__ x,
                                         double* __restrict__ d, double* __restrict__ negj) {
#ifdef FO_LINK_GENERATED
  fo_gen_jac(negj - p.sl.negj * ln.L + ln.lane, TEAM_W, TEAM_N, p.o.gen_index);
#else
  constexpr int kBatch = 8;
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n, R = p.t.R, P = p.t.P;
  const double* __restrict__ kc = p.k + ln.cell * p.kcs;
#pragma unroll 4
  for (int j = 0; j < R; ++j) {
    const double kj = __ldg(kc + (int64_t)j * p.krs);
    for (int a = 0; a < P; ++a) {
      double prod = kj;
      for (int q = 0; q < P; ++q) {
        if (q == a) continue;
        int s = __ldg(p.t.react + j * P + q);
        if (s != n) prod = __dmul_rn(prod, SCR(x, s));
      }
      SCR(d, j * P + a) = prod;
    }
  }
  for (int e = 0; e < p.t.nnzj; ++e) {
    double acc = 0.0;
    const int t1 = __ldg(p.t.jt_ptr + e + 1);
    int t = __ldg(p.t.jt_ptr + e);
    for (; t + kBatch <= t1; t += kBatch) {
      double v[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) v[b] = SCR(d, __ldg(p.t.jt_idx + t + b));
#pragma unroll
      for (int b = 0; b < kBatch; ++b) acc = __dadd_rn(acc, __dmul_rn(__ldg(p.t.jt_val + t + b), v[b]));
    }
    for (; t < t1; ++t) acc = __dadd_rn(acc, __dmul_rn(__ldg(p.t.jt_val + t), SCR(d, __ldg(p.t.jt_idx + t))));
    SCR(negj, e) = acc;
  }
#endif
}

// Row r of the stage matrix alpha*M - J scattered into the dense work row w
// over the row's filled pattern (fastode/linalg.py:60-67). With alg_only,
// the projection's matrix diag(M) - J with the differential rows of J
// dropped (fastode/linalg.py:62-63, alpha = 1).
__device__ __forceinline__ void assemble_row(const SolveParams& p, const Lane& ln, int r, int q0, int q1,
                                             double alpha, const double* negj, double* w, bool alg_only) {
  const int L = ln.L, lane = ln.lane;
  const int32_t* __restrict__ col = p.t.lu_col;
  for (int q = q0; q < q1; ++q) WROW(__ldg(col + q)) = 0.0;
  const double mr = __ldg(p.t.mass + r);
  if (!alg_only || mr == 0.0) {
    const int e1 = __ldg(p.t.j_row_ptr + r + 1);
    for (int e = __ldg(p.t.j_row_ptr + r); e < e1; ++e) WROW(__ldg(p.t.j_col + e)) = SCR(negj, e);
  }
  WROW(r) = __dadd_rn(WROW(r), __dmul_rn(alpha, mr));
}

// In-place pivot-free LU of alpha*M - J on the precomputed fill pattern,
// row by row (up-looking). Row r is scattered into the dense work row w,
// eliminated with the finished rows above it, and gathered back. The
// diagonal slot keeps the reciprocal of the pivot. Replaces SuperLU's gstrf
// (fastode/linalg.py:70-78) and LAPACK getrf (fastode/linalg.py:15-18).
__device__ __noinline__ void factor(const SolveParams& p, const Lane& ln, double alpha, const double* negj, double* lu,
                       double* w, bool alg_only) {
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n;
  const int32_t* __restrict__ rowp = p.t.lu_row_ptr;
  const int32_t* __restrict__ diag = p.t.lu_diag;
  const int32_t* __restrict__ col = p.t.lu_col;
  for (int r = 0; r < n; ++r) {
    const int q0 = __ldg(rowp + r), q1 = __ldg(rowp + r + 1), dg = __ldg(diag + r);
    assemble_row(p, ln, r, q0, q1, alpha, negj, w, alg_only);
    for (int q = q0; q < dg; ++q) {
      const int k = __ldg(col + q);
      const double l = WROW(k) * SCR(lu, __ldg(diag + k));
      SCR(lu, q) = l;
      const int u1 = __ldg(rowp + k + 1);
      int u = __ldg(diag + k) + 1;
      for (; u + 3 < u1; u += 4) {
        const int c0 = __ldg(col + u), c1 = __ldg(col + u + 1), c2 = __ldg(col + u + 2), c3 = __ldg(col + u + 3);
        const double v0 = SCR(lu, u), v1 = SCR(lu, u + 1), v2 = SCR(lu, u + 2), v3 = SCR(lu, u + 3);
        WROW(c0) = fma(-l, v0, WROW(c0));
        WROW(c1) = fma(-l, v1, WROW(c1));
        WROW(c2) = fma(-l, v2, WROW(c2));
        WROW(c3) = fma(-l, v3, WROW(c3));
      }
      for (; u < u1; ++u) {
        const int c = __ldg(col + u);
        WROW(c) = fma(-l, SCR(lu, u), WROW(c));
      }
    }
    SCR(lu, dg) = 1.0 / WROW(r);
    for (int q = dg + 1; q < q1; ++q) SCR(lu, q) = WROW(__ldg(col + q));
  }
}

// The same factorization driven by the precomputed elimination stream
// (symbolic.h): every row's multipliers and updates are one flat sequence of
// (x, y) entries in chunks of kChunk. The work row is compressed to the row's
// own pattern (w[y] stands for lu[row start + y]), which leaves room in shared
// memory for a ring of kRingChunks chunks: each lane copies its own 8-byte U
// entries (of finished rows, or pivot reciprocals — nothing the row writes)
// into the ring with cp.async several chunks ahead of their use, so a warp
// keeps up to (kRingChunks - 1) * kChunk 256-byte loads in flight without
// holding them in registers.
constexpr int kChunk = kStreamChunk;

// Stream metadata, packed to 32 bits per entry: (position << 16) | slot, slot
// bit 15 marking a multiplier, slot 0x7fff padding. A chunk is four uint4.
struct Meta {
  uint4 q[kChunk / 4];
};

__device__ __forceinline__ void meta_load(const uint32_t* __restrict__ m, Meta& out) {
#pragma unroll
  for (int i = 0; i < kChunk / 4; ++i) out.q[i] = __ldg(reinterpret_cast<const uint4*>(m) + i);
}

__device__ __forceinline__ uint32_t meta_at(const Meta& m, int s) {
  const uint4 v = m.q[s >> 2];
  return (s & 3) == 0 ? v.x : (s & 3) == 1 ? v.y : (s & 3) == 2 ? v.z : v.w;
}

// Copy the chunk's 16 operands of this lane (U entries of finished rows or
// pivot reciprocals; padding copies entry 0) into the ring slot.
__device__ __forceinline__ void ring_issue(const Meta& m, const double* __restrict__ lu, int L, int lane,
                                           double* ring_slot) {
  const unsigned dst0 = (unsigned)__cvta_generic_to_shared(ring_slot + lane);
#pragma unroll
  for (int s = 0; s < kChunk; ++s) {
    const uint32_t word = meta_at(m, s);
    const double* g = lu + (int64_t)(word >> 16) * L + lane;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst0 + (unsigned)(s * L * 8)), "l"(g));
  }
}

__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__device__ __forceinline__ void ring_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kRingChunks - 1) : "memory");
}

// A hazard-free chunk (symbolic.cpp builds them) in three parts: read every
// work-row value the chunk touches, apply its multipliers and updates in order
// in registers (updates are independent FMAs; only a multiplier starts a new
// dependency), and write the updated values back. The factorization writes a
// chunk back only after the next chunk has read its values and issued its
// FMAs, which the two-chunk hazard rule makes safe.
__device__ __forceinline__ void chunk_read(const Meta& m, const double* w, int L, int lane, double (&wv)[kChunk]) {
#pragma unroll
  for (int s = 0; s < kChunk; ++s) {
    const uint32_t y = meta_at(m, s) & 0x7fffu;
    wv[s] = y != 0x7fffu ? WROW(y) : 0.0;
  }
}

__device__ __forceinline__ void chunk_fma(const Meta& m, const double* ring_slot, double* lu, int L, int lane,
                                          double (&wv)[kChunk], double& l, int& q) {
#pragma unroll
  for (int s = 0; s < kChunk; ++s) {
    const uint32_t word = meta_at(m, s);
    const uint32_t y = word & 0x7fffu;
    const double v = ring_slot[s * L + lane];
    if (word & 0x8000u) {
      l = wv[s] * v;
      SCR(lu, q) = l;
      ++q;
    } else if (y != 0x7fffu) {
      wv[s] = fma(-l, v, wv[s]);
    }
  }
}

__device__ __forceinline__ void chunk_write(const Meta& m, double* w, int L, int lane, const double (&wv)[kChunk]) {
#pragma unroll
  for (int s = 0; s < kChunk; ++s) {
    const uint32_t word = meta_at(m, s);
    const uint32_t y = word & 0x7fffu;
    if (!(word & 0x8000u) && y != 0x7fffu) WROW(y) = wv[s];
  }
}

template <int kL>
__device__ __noinline__ void factor_stream(const SolveParams& p, const Lane& ln, double alpha, const double* negj,
                                           double* lu, double* w, bool alg_only) {
  const int L = kL ? kL : ln.L, lane = ln.lane;
  const int n = p.t.n;
  const int32_t* __restrict__ rowp = p.t.lu_row_ptr;
  const int32_t* __restrict__ diag = p.t.lu_diag;
  double* ring = w + (int64_t)p.t.max_row_len * L;
  for (int r = 0; r < n; ++r) {
    const int q0 = __ldg(rowp + r), q1 = __ldg(rowp + r + 1), dg = __ldg(diag + r);
    // assemble row r of alpha*M - J into the compressed work row
    for (int s = 0; s < q1 - q0; ++s) WROW(s) = 0.0;
    const double mr = __ldg(p.t.mass + r);
    if (!alg_only || mr == 0.0) {
      const int e1 = __ldg(p.t.j_row_ptr + r + 1);
      for (int e = __ldg(p.t.j_row_ptr + r); e < e1; ++e) WROW(__ldg(p.t.j_pos + e) - q0) = SCR(negj, e);
    }
    WROW(dg - q0) = __dadd_rn(WROW(dg - q0), __dmul_rn(alpha, mr));
    const int t0 = __ldg(p.t.el_ptr + r);
    const int nch = (__ldg(p.t.el_ptr + r + 1) - t0) / kChunk;
    const uint32_t* meta = p.t.elp + t0;
    double l = 0.0;
    int q = q0;
    Meta mi, mc;
#pragma unroll 1
    for (int c = 0; c < kRingChunks - 1; ++c) {
      if (c < nch) {
        meta_load(meta + c * kChunk, mi);
        ring_issue(mi, lu, L, lane, ring + (int64_t)(c % kRingChunks) * kChunk * L);
      }
      ring_commit();
    }
    if (kRingChunks - 1 < nch) meta_load(meta + (kRingChunks - 1) * kChunk, mi);
    if (nch > 0) meta_load(meta, mc);
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
      const int ahead = c + kRingChunks - 1;
      Meta mi_next, mc_next;
      if (ahead + 1 < nch) meta_load(meta + (ahead + 1) * kChunk, mi_next);
      if (c + 1 < nch) meta_load(meta + (c + 1) * kChunk, mc_next);
      if (ahead < nch) ring_issue(mi, lu, L, lane, ring + (int64_t)(ahead % kRingChunks) * kChunk * L);
      ring_commit();
      ring_wait();
      double wc[kChunk];
      chunk_read(mc, w, L, lane, wc);
      chunk_fma(mc, ring + (int64_t)(c % kRingChunks) * kChunk * L, lu, L, lane, wc, l, q);
      chunk_write(mc, w, L, lane, wc);
      mi = mi_next;
      mc = mc_next;
    }
    SCR(lu, dg) = 1.0 / WROW(dg - q0);
    for (int qq = dg + 1; qq < q1; ++qq) SCR(lu, qq) = WROW(qq - q0);
  }
}

// ---- the compact factorization (FO_VARIANT_COMPACT) ------------------------------
//
// Row r is eliminated in two passes over halves of its slots (symbolic.h):
// pass A is the elimination restricted to the row's leading columns and
// stores its multipliers as it makes them; pass B applies every multiplier's
// updates of the trailing columns, in the same order, reloading A's
// multipliers from the LU storage through the same ring as the U operands (a
// block-scope fence between the passes orders this thread's stores of them
// before the asynchronous copies that read them back). The work row therefore
// holds half a row, and the factors are the pipelined ones bit for bit. The
// operands are staged one chunk ahead in a two-slot ring: with twice as many
// groups resident per SM, a deeper ring buys nothing.

template <int kL>
__device__ __noinline__ void factor_compact(const SolveParams& p, const Lane& ln, double alpha, const double* negj,
                                            double* lu, double* w, bool alg_only) {
  const int L = kL ? kL : ln.L, lane = ln.lane;
  const int n = p.t.n;
  const int32_t* __restrict__ rowp = p.t.lu_row_ptr;
  const int32_t* __restrict__ diag = p.t.lu_diag;
  double* ring = w + (int64_t)p.t.cmax_half * L;
  for (int r = 0; r < n; ++r) {
    const int q0 = __ldg(rowp + r), len = __ldg(rowp + r + 1) - q0, dslot = __ldg(diag + r) - q0;
    const int split = __ldg(p.t.cs_split + r), jsplit = __ldg(p.t.cs_jsplit + r);
    const double mr = __ldg(p.t.mass + r);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const int base = pass ? split : 0, cnt = pass ? len - split : split;
      for (int s = 0; s < cnt; ++s) WROW(s) = 0.0;
      if (!alg_only || mr == 0.0) {
        const int e0 = pass ? jsplit : __ldg(p.t.j_row_ptr + r);
        const int e1 = pass ? __ldg(p.t.j_row_ptr + r + 1) : jsplit;
        for (int e = e0; e < e1; ++e) WROW(__ldg(p.t.j_pos + e) - q0 - base) = SCR(negj, e);
      }
      const bool has_diag = dslot >= base && dslot < base + cnt;
      if (has_diag) WROW(dslot - base) = __dadd_rn(WROW(dslot - base), __dmul_rn(alpha, mr));
      const int t0 = __ldg(p.t.ce_ptr + 2 * r + pass);
      const int nch = (__ldg(p.t.ce_ptr + 2 * r + pass + 1) - t0) / kChunk;
      const uint32_t* meta = p.t.cep + t0;
      double* qlu = lu + (int64_t)(q0 + base) * L;     // this pass's slot s stands for lu[q0 + base + s]
      double l = 0.0;
      Meta mc, mi;
      if (pass) __threadfence_block();   // pass A's stores before pass B's copies read them
      if (nch > 0) {
        meta_load(meta, mc);
        ring_issue(mc, lu, L, lane, ring);
      }
      ring_commit();
      if (nch > 1) meta_load(meta + kChunk, mi);
#pragma unroll 1
      for (int c = 0; c < nch; ++c) {
        Meta mn;
        if (c + 2 < nch) meta_load(meta + (c + 2) * kChunk, mn);
        if (c + 1 < nch) ring_issue(mi, lu, L, lane, ring + (int64_t)((c + 1) % kCompactRing) * kChunk * L);
        ring_commit();
        asm volatile("cp.async.wait_group %0;" ::"n"(kCompactRing - 1) : "memory");
        const double* rs = ring + (int64_t)(c % kCompactRing) * kChunk * L;
        double wv[kChunk];
#pragma unroll
        for (int s = 0; s < kChunk; ++s) {
          const uint32_t y = meta_at(mc, s) & 0x7fffu;
          wv[s] = y < kReloadSlot ? WROW(y) : 0.0;
        }
#pragma unroll
        for (int s = 0; s < kChunk; ++s) {
          const uint32_t word = meta_at(mc, s);
          const uint32_t y = word & 0x7fffu;
          if (word & 0x8000u) {
            l = wv[s] * rs[s * L + lane];
            SCR(qlu, y) = l;
          } else if (y == kReloadSlot) {
            l = rs[s * L + lane];
          } else if (y != 0x7fffu) {
            wv[s] = fma(-l, rs[s * L + lane], wv[s]);
          }
        }
#pragma unroll
        for (int s = 0; s < kChunk; ++s) {
          const uint32_t word = meta_at(mc, s);
          const uint32_t y = word & 0x7fffu;
          if (!(word & 0x8000u) && y < kReloadSlot) WROW(y) = wv[s];
        }
        mc = mi;
        mi = mn;
      }
      if (has_diag) WROW(dslot - base) = 1.0 / WROW(dslot - base);
      for (int s = dslot > base ? dslot - base : 0; s < cnt; ++s) SCR(qlu, s) = WROW(s);
    }
  }
}

// Forward and backward substitution driven by the solve streams
// (symbolic.h): a chunk's metadata is loaded two chunks ahead of its use and
// its factor entries one chunk ahead (neither depends on the solution), so the
// entries' loads never wait for their positions; the solution entries are read
// from shared memory when the chunk computes. kMixed: an operand may lie in
// the other, finished half of the vector in global memory (kGlobalOperand).
template <bool kMixed>
__device__ __forceinline__ void solve_values(const int4 (&m)[kChunk / 2], const double* __restrict__ lu,
                                             const double* xg, int L, int lane, double (&v)[kChunk],
                                             double (&g)[kChunk]) {
#pragma unroll
  for (int s = 0; s < kChunk / 2; ++s) {
    const int p0 = m[s].x >= 0 ? m[s].x : -1 - m[s].x;
    const int p1 = m[s].z >= 0 ? m[s].z : -1 - m[s].z;
    v[2 * s] = lu[(int64_t)p0 * L + lane];
    v[2 * s + 1] = lu[(int64_t)p1 * L + lane];
    if (kMixed) {
      const int y0 = m[s].y, y1 = m[s].w;
      g[2 * s] = (y0 >= 0 && (y0 & kGlobalOperand)) ? xg[(int64_t)(y0 & ~kGlobalOperand) * L + lane] : 0.0;
      g[2 * s + 1] = (y1 >= 0 && (y1 & kGlobalOperand)) ? xg[(int64_t)(y1 & ~kGlobalOperand) * L + lane] : 0.0;
    }
  }
}

__device__ __forceinline__ void solve_meta(const int2* __restrict__ meta, int4 (&m)[kChunk / 2]) {
#pragma unroll
  for (int s = 0; s < kChunk / 2; ++s) m[s] = __ldg(reinterpret_cast<const int4*>(meta) + s);
}

// Two partial sums per row, entry s of a chunk feeding sum s mod 2: the row's
// FMAs form two independent chains. More sums hide more FP64 latency but cost
// registers the chunk buffers need (measured per interval: four sums 4.5%
// slower, eight 10% slower).
template <bool kBackward, bool kMixed>
__device__ __forceinline__ void solve_entry(int s, int y, double v, double gv, double* w, int L, int lane,
                                            double (&acc)[2]) {
  if (y >= 0) {
    const double x = (kMixed && (y & kGlobalOperand)) ? gv : WROW(y);
    acc[s & 1] = fma(-v, x, acc[s & 1]);
  } else if (y != kNoop) {
    const int r = -1 - y;
    const double b = WROW(r) + (acc[0] + acc[1]);
    WROW(r) = kBackward ? b * v : b;
    acc[0] = acc[1] = 0.0;
  }
}

template <bool kBackward, bool kMixed>
__device__ __forceinline__ void solve_compute(const int4 (&m)[kChunk / 2], const double (&v)[kChunk],
                                              const double (&g)[kChunk], double* w, int L, int lane, double (&acc)[2]) {
#pragma unroll
  for (int s = 0; s < kChunk / 2; ++s) {
    solve_entry<kBackward, kMixed>(2 * s, m[s].y, v[2 * s], g[2 * s], w, L, lane, acc);
    solve_entry<kBackward, kMixed>(2 * s + 1, m[s].w, v[2 * s + 1], g[2 * s + 1], w, L, lane, acc);
  }
}

// kMixed: the stream's operands may lie in xg (kGlobalOperand set).
template <bool kBackward, bool kMixed = false>
__device__ __forceinline__ void solve_stream(const int2* __restrict__ st, int nst, const double* lu, double* w, int L,
                                             int lane,
                             const double* xg = nullptr) {
  int4 mc[kChunk / 2], mn[kChunk / 2];
  double vc[kChunk], gc[kChunk];
  double acc[2] = {0.0, 0.0};
  const int nch = nst / kChunk;
  if (nch == 0) return;            // an empty half (a one-species system)
  solve_meta(st, mc);
  solve_values<kMixed>(mc, lu, xg, L, lane, vc, gc);
  if (nch > 1) solve_meta(st + kChunk, mn);
#pragma unroll 1
  for (int c = 0; c < nch; ++c) {
    int4 mnn[kChunk / 2];
    double vn[kChunk], gn[kChunk];
    if (c + 1 < nch) solve_values<kMixed>(mn, lu, xg, L, lane, vn, gn);
    if (c + 2 < nch) solve_meta(st + (c + 2) * kChunk, mnn);
    solve_compute<kBackward, kMixed>(mc, vc, gc, w, L, lane, acc);
#pragma unroll
    for (int s = 0; s < kChunk / 2; ++s) {
      mc[s] = mn[s];
      mn[s] = mnn[s];
    }
#pragma unroll
    for (int s = 0; s < kChunk; ++s) {
      vc[s] = vn[s];
      gc[s] = gn[s];
    }
  }
}

template <int kL>
__device__ __noinline__ void lu_solve_pipelined(const SolveParams& p, const Lane& ln, const double* lu, double* w) {
  const int L = kL ? kL : ln.L;
  solve_stream<false>(p.t.sf, p.t.nsf, lu, w, L, ln.lane);
  solve_stream<true>(p.t.sb, p.t.nsb, lu, w, L, ln.lane);
}

// The compact solves: b and x are per-lane vectors in global memory (they may
// alias) and shared memory holds one half of the vector at a time. Forward
// over rows [0, csm) needs only that half; the finished half is stored, and
// forward over rows [csm, n) then reads it from x, as does nothing else until
// backward over rows [n-1, csm) has finished the second half, which is stored
// for backward over rows [csm-1, 0) to read.
template <int kL>
__device__ __noinline__ void lu_solve_compact_l(const SolveParams& p, const Lane& ln, const double* lu, double* w,
                                                const double* b, double* x) {
  const int L = kL ? kL : ln.L, lane = ln.lane;
  const int n = p.t.n, m = p.t.csm;
  for (int i = 0; i < m; ++i) WROW(i) = SCR(b, i);
  solve_stream<false>(p.t.csf_a, p.t.ncsf_a, lu, w, L, lane);
  for (int i = 0; i < m; ++i) SCR(x, i) = WROW(i);
  for (int i = m; i < n; ++i) WROW(i - m) = SCR(b, i);
  solve_stream<false, true>(p.t.csf_b, p.t.ncsf_b, lu, w, L, lane, x);
  solve_stream<true>(p.t.csb_b, p.t.ncsb_b, lu, w, L, lane);
  for (int i = m; i < n; ++i) SCR(x, i) = WROW(i - m);
  for (int i = 0; i < m; ++i) WROW(i) = SCR(x, i);
  solve_stream<true, true>(p.t.csb_a, p.t.ncsb_a, lu, w, L, lane, x);
  for (int i = 0; i < m; ++i) SCR(x, i) = WROW(i);
}

// The stream kernels specialised for 32 lanes (one warp per group, the usual
// launch) fold the lane stride into immediate offsets; other group sizes run
// the general instantiation.
__device__ __forceinline__ void lu_solve_compact(const SolveParams& p, const Lane& ln, const double* lu, double* w,
                                                 const double* b, double* x) {
  if (ln.L == 32) lu_solve_compact_l<32>(p, ln, lu, w, b, x);
  else lu_solve_compact_l<0>(p, ln, lu, w, b, x);
}

// Forward and backward substitution in place on w (fastode/linalg.py:80-81),
// each row's terms in the order in which their values finish: ascending
// columns forward, descending columns backward (the generated solves' order,
// which lets a finished value update every remaining row at once).
__device__ void lu_solve(const SolveParams& p, const Lane& ln, const double* lu, double* w) {
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n;
  const int32_t* __restrict__ rowp = p.t.lu_row_ptr;
  const int32_t* __restrict__ diag = p.t.lu_diag;
  const int32_t* __restrict__ col = p.t.lu_col;
  for (int r = 0; r < n; ++r) {
    double acc = WROW(r);
    const int dg = __ldg(diag + r);
    for (int q = __ldg(rowp + r); q < dg; ++q) acc = fma(-SCR(lu, q), WROW(__ldg(col + q)), acc);
    WROW(r) = acc;
  }
  for (int r = n - 1; r >= 0; --r) {
    double acc = WROW(r);
    const int dg = __ldg(diag + r);
    for (int q = __ldg(rowp + r + 1) - 1; q > dg; --q) acc = fma(-SCR(lu, q), WROW(__ldg(col + q)), acc);
    WROW(r) = acc * SCR(lu, dg);
  }
}

// The generated variant (FO_VARIANT_GENERATED) exists only in the kernels
// linked per mechanism with the generated functions.
// Those kernels run nothing else (the launch code guarantees the variant),
// so the other variants' factorizations and solves are not compiled into
// them.
__device__ __forceinline__ bool generated(const SolveParams&) {
#ifdef FO_LINK_GENERATED
  return true;
#else
  return false;
#endif
}

// The variants that solve a per-lane vector in place rather than the work row.
__device__ __forceinline__ bool solves_in_place(const SolveParams& p) {
  return p.o.variant == FO_VARIANT_COMPACT || generated(p);
}

#ifdef FO_LINK_GENERATED
// The dense square's elimination (GenLayout): nb x nb blocks of kDenseBlock
// rows and columns in tile-major order, `a` this lane's first item. A warp
// holds a block in registers while it takes the updates of earlier pivots, two
// columns of operands in flight (36 DFMAs per 12 loads). Each entry receives
// its updates in ascending pivot order, as in the row-by-row elimination. The
// loops are a few kilobytes of code, so the warps of an SM share them in the
// instruction cache wherever each of them is.
constexpr int kDB = kDenseBlock;

__device__ __forceinline__ double* dense_block(double* a, int nb, int bi, int bj) {
  return a + (int64_t)(bi * nb + bj) * kDB * kDB * 32;
}

__device__ __forceinline__ void block_load(const double* t, double (&c)[kDB][kDB]) {
#pragma unroll
  for (int i = 0; i < kDB; ++i)
#pragma unroll
    for (int j = 0; j < kDB; ++j) c[i][j] = t[(i * kDB + j) * 32];
}

__device__ __forceinline__ void block_store(double* t, const double (&c)[kDB][kDB]) {
#pragma unroll
  for (int i = 0; i < kDB; ++i)
#pragma unroll
    for (int j = 0; j < kDB; ++j) t[(i * kDB + j) * 32] = c[i][j];
}

// c -= sum over m blocks of L(bi, .) U(., bj); ustep: doubles between U blocks
__device__ __forceinline__ void block_update(double (&c)[kDB][kDB], const double* l, const double* u, int m,
                                             int64_t ustep) {
  double a[2][kDB], b[2][kDB];
  if (m == 0) return;
#pragma unroll
  for (int i = 0; i < kDB; ++i) {
    a[0][i] = l[i * kDB * 32];
    b[0][i] = u[i * 32];
  }
#pragma unroll 1
  for (int q = 0; q < m; ++q) {
    const bool more = q + 1 < m;
    const double* ln = more ? l + kDB * kDB * 32 : l;   // the last pivot's lookahead rereads
    const double* un = more ? u + ustep : u;
#pragma unroll
    for (int k = 0; k < kDB; ++k) {
      const double* lk = k + 1 < kDB ? l + (k + 1) * 32 : ln;
      const double* uk = k + 1 < kDB ? u + (k + 1) * kDB * 32 : un;
#pragma unroll
      for (int i = 0; i < kDB; ++i) {
        a[(k + 1) & 1][i] = lk[i * kDB * 32];
        b[(k + 1) & 1][i] = uk[i * 32];
      }
#pragma unroll
      for (int i = 0; i < kDB; ++i)
#pragma unroll
        for (int j = 0; j < kDB; ++j) c[i][j] = fma(-a[k & 1][i], b[k & 1][j], c[i][j]);
    }
    l = ln;
    u = un;
  }
}

// The step's own pivots on a block below (left) or right of the diagonal
// block d: multipliers and their updates, or the updates of its rows.
__device__ __forceinline__ void block_finish(double (&c)[kDB][kDB], const double* d, bool left) {
#pragma unroll
  for (int k = 0; k < kDB; ++k) {
    if (left) {
      const double rk = d[(k * kDB + k) * 32];
#pragma unroll
      for (int i = 0; i < kDB; ++i) c[i][k] *= rk;
#pragma unroll
      for (int j = k + 1; j < kDB; ++j) {
        const double u = d[(k * kDB + j) * 32];
#pragma unroll
        for (int i = 0; i < kDB; ++i) c[i][j] = fma(-c[i][k], u, c[i][j]);
      }
    } else {
#pragma unroll
      for (int i = k + 1; i < kDB; ++i) {
        const double m = d[(i * kDB + k) * 32];
#pragma unroll
        for (int j = 0; j < kDB; ++j) c[i][j] = fma(-m, c[k][j], c[i][j]);
      }
    }
  }
}

// The diagonal block's own pivots.
__device__ __forceinline__ void block_factor(double (&c)[kDB][kDB]) {
#pragma unroll
  for (int k = 0; k < kDB; ++k) {
    const double rk = 1.0 / c[k][k];
    c[k][k] = rk;
#pragma unroll
    for (int i = k + 1; i < kDB; ++i) {
      c[i][k] *= rk;
#pragma unroll
      for (int j = k + 1; j < kDB; ++j) c[i][j] = fma(-c[i][k], c[k][j], c[i][j]);
    }
  }
}

// A team, right-looking. Step s updates every block that remains with the
// pivots of the block before it, one warp per block, and the warp of the
// diagonal block factors that; after a barrier the others of its row and column
// take the step's own pivots. A sub-partition issues one DFMA in 64 cycles or
// more whichever of its warps it comes from, so what counts is how evenly a
// step's blocks fill four sub-partitions: left-looking the last steps have 1,
// 3, 5, ... blocks, with the most updates each, and the 506 updates of 12 x 12
// blocks take the time of 644. 4,096 cells of 210/500, recorded and reversed
// (one team of 16 per SM): 180.6 ms left-looking, 172.4 right-looking. Panels of
// two pivot blocks, which load and store a block half as often, gain nothing
// beyond the runs' spread. With and without them, ms: the same adjoint 168.2 and
// 169.5 (runs of one side differ by 0.9%), three host intervals of 8,192 cells of
// 120/260 9.02 and 8.94, two intervals of TS1 on 8,200 cells 7.75 and 7.68, one
// 210/500 group on a cluster 27.3 and 25.5.
__device__ __noinline__ void dense_lu_team(double* a, int nb) {
  const int64_t ustep = (int64_t)nb * kDB * kDB * 32;
  const int w = TEAM_W, wn = TEAM_N;
#pragma unroll 1
  for (int s = 0; s < nb; ++s) {
    const int m = nb - s, count = s > 0 ? m * m : 1, before = s > 0 ? s - 1 : 0;
#pragma unroll 1
    for (int q = w; q < count; q += wn) {
      const int bi = s + q / m, bj = s + q % m;
      double* t = dense_block(a, nb, bi, bj);
      double c[kDB][kDB];
      block_load(t, c);
      block_update(c, dense_block(a, nb, bi, before), dense_block(a, nb, before, bj), s - before, ustep);
      if (q == 0) block_factor(c);
      block_store(t, c);
    }
    team_sync();
    const int rest = 2 * (m - 1);
    const double* d = dense_block(a, nb, s, s);
#pragma unroll 1
    for (int q = w; q < rest; q += wn) {
      const int k = s + 1 + q / 2;
      const bool left = (q & 1) != 0;
      double* t = dense_block(a, nb, left ? k : s, left ? s : k);
      double c[kDB][kDB];
      block_load(t, c);
      block_finish(c, d, left);
      block_store(t, c);
    }
    if (rest > 0) team_sync();
  }
}

// One warp alone, left-looking: a block takes all its updates and its own
// step's pivots in registers, in one pass over the square.
__device__ __noinline__ void dense_lu_warp(double* a, int nb) {
  const int64_t ustep = (int64_t)nb * kDB * kDB * 32;
#pragma unroll 1
  for (int s = 0; s < nb; ++s) {
    // block 0 of the step is the diagonal one, 2m - 1 and 2m those m below
    // and m right of it
    const double* d = dense_block(a, nb, s, s);
#pragma unroll 1
    for (int q = 0; q < 2 * (nb - s) - 1; ++q) {
      const int m = s + (q + 1) / 2;
      const bool left = (q & 1) != 0;
      const int bi = left ? m : s, bj = left ? s : m;
      double* t = dense_block(a, nb, bi, bj);
      double c[kDB][kDB];
      block_load(t, c);
      block_update(c, dense_block(a, nb, bi, 0), dense_block(a, nb, 0, bj), s, ustep);
      if (q == 0) block_factor(c);
      else block_finish(c, d, left);
      block_store(t, c);
    }
  }
}

__device__ __forceinline__ void dense_lu(double* a, int nb) {
  if (TEAM_N == 1) dense_lu_warp(a, nb);
  else dense_lu_team(a, nb);
}
#endif

#ifdef FO_LINK_GENERATED
// One triangle of the square's solves in place on its part of the solve vector
// (x, this lane's first item): blocks of kDB rows finish in ascending order
// (kUp) or descending order, each row subtracting entry(i, k) x_k as its
// values finish and then, kScale, taking the diagonal item (1 / pivot);
// kTransposed: entry(i, k) is the stored (k, i). Warp w of wn (one block's
// warps: a triangle is a chain of small steps) updates every wn-th block that
// remains with the block just finished; the warp of the next block finishes it
// too, so a step has one barrier. One warp alone sums a block's terms in
// registers instead. As straight-line code a triangle of 72 rows was 0.6 MB,
// fetched anew by every solve.
template <bool kUp, bool kScale, bool kTransposed>
__device__ __noinline__ void square_triangle(const double* a, double* x, int nb, int w, int wn) {
  // c_i -= sum of entry(i, k) v_k over a whole block (block b's rows, block k's columns)
  auto update = [&](double (&c)[kDB], int b, int k) {
    const double* t = a + (int64_t)(kTransposed ? k * nb + b : b * nb + k) * kDB * kDB * 32;
    const double* xk = x + (int64_t)k * kDB * 32;
    double v[kDB], e[kDB][kDB];
#pragma unroll
    for (int q = 0; q < kDB; ++q) v[q] = xk[q * 32];
#pragma unroll
    for (int i = 0; i < kDB; ++i)
#pragma unroll
      for (int q = 0; q < kDB; ++q) e[i][q] = t[(kTransposed ? q * kDB + i : i * kDB + q) * 32];
#pragma unroll
    for (int m = 0; m < kDB; ++m) {
      const int q = kUp ? m : kDB - 1 - m;
#pragma unroll
      for (int i = 0; i < kDB; ++i) c[i] = fma(-e[i][q], v[q], c[i]);
    }
  };
  auto finish = [&](double (&c)[kDB], int b) {
    const double* t = a + (int64_t)(b * nb + b) * kDB * kDB * 32;
#pragma unroll
    for (int m = 0; m < kDB; ++m) {
      const int q = kUp ? m : kDB - 1 - m;
      if (kScale) c[q] *= t[(q * kDB + q) * 32];
#pragma unroll
      for (int i = 0; i < kDB; ++i)
        if (kUp ? i > q : i < q) c[i] = fma(-t[(kTransposed ? q * kDB + i : i * kDB + q) * 32], c[q], c[i]);
    }
  };
  auto load = [&](double (&c)[kDB], int b) {
#pragma unroll
    for (int i = 0; i < kDB; ++i) c[i] = x[(int64_t)(b * kDB + i) * 32];
  };
  auto store = [&](const double (&c)[kDB], int b) {
#pragma unroll
    for (int i = 0; i < kDB; ++i) x[(int64_t)(b * kDB + i) * 32] = c[i];
  };
  if (wn == 1) {
#pragma unroll 1
    for (int m = 0; m < nb; ++m) {
      const int b = kUp ? m : nb - 1 - m;
      double c[kDB];
      load(c, b);
#pragma unroll 1
      for (int q = 0; q < m; ++q) update(c, b, kUp ? q : nb - 1 - q);
      finish(c, b);
      store(c, b);
    }
    return;
  }
#pragma unroll 1
  for (int m = -1; m < nb - 1; ++m) {
    // block m (in finishing order) is done; those after it take its terms
    const int k = kUp ? m : nb - 1 - m;
#pragma unroll 1
    for (int r = m + 1 + w; r < (m < 0 ? 1 : nb); r += wn) {
      const int b = kUp ? r : nb - 1 - r;
      double c[kDB];
      load(c, b);
      if (m >= 0) update(c, b, k);
      if (r == m + 1) finish(c, b);
      store(c, b);
    }
    __syncthreads();
  }
}

// x = A^-1 b or A^-T b in place on the solve vector, by the warps of a block;
// the factors are the stage matrix's or, kProjection, the projection's. Every
// warp's right-hand side is in place on entry (the phases begin and end with
// the barrier of `wn` warps).
template <bool kTransposed, bool kProjection>
__device__ __forceinline__ void generated_solve(const SolveParams& p, double* base, int w, int wn) {
  const int mech = p.o.gen_index, nb = kProjection ? 0 : p.sl.nb;
  if (kProjection) {
    if (kTransposed) fo_gen_solve_t_p_up(base, w, wn, mech);
    else fo_gen_solve_p_up(base, w, wn, mech);
  } else {
    if (kTransposed) fo_gen_solve_t_up(base, w, wn, mech);
    else fo_gen_solve_up(base, w, wn, mech);
  }
  if (nb > 0) {
    const double* a = base + p.sl.dn * 32;
    double* x = base + (p.sl.xs + p.t.n - (int64_t)nb * kDB) * 32;
    square_triangle<true, kTransposed, kTransposed>(a, x, nb, w, wn);
    square_triangle<false, !kTransposed, kTransposed>(a, x, nb, w, wn);
  }
  if (kProjection) {
    if (kTransposed) fo_gen_solve_t_p_down(base, w, wn, mech);
    else fo_gen_solve_p_down(base, w, wn, mech);
  } else {
    if (kTransposed) fo_gen_solve_t_down(base, w, wn, mech);
    else fo_gen_solve_down(base, w, wn, mech);
  }
}

// x = A^-1 b in place on the solve vector by the whole team. A solve is a chain
// of small steps: one block of a cluster with its own barriers and L1 is
// faster than all of them (a solve of 210/500: 0.32 M cycles and 0.38 M).
template <bool kProjection>
__device__ __forceinline__ void team_solve(const SolveParams& p, double* base) {
  if (cluster_team()) {
    team_sync();   // the right-hand side, from every block
    if (cluster_rank() == 0) generated_solve<false, kProjection>(p, base, BLOCK_W, BLOCK_N);
    team_sync();
  } else {
    generated_solve<false, kProjection>(p, base, BLOCK_W, BLOCK_N);
  }
}
#endif

__device__ void factor_any(const SolveParams& p, const Lane& ln, double alpha, const double* negj, double* lu,
                           double* w, bool alg_only) {
#ifdef FO_LINK_GENERATED
  double* base = lu - p.sl.lu * ln.L + ln.lane;
  if (alg_only) {
    fo_gen_factor_p(base, TEAM_W, TEAM_N, p.o.gen_index);
  } else {
    fo_gen_factor(base, alpha, TEAM_W, TEAM_N, p.o.gen_index);
    if (p.sl.nb > 0) {
      dense_lu(base + p.sl.dn * ln.L, p.sl.nb);
    }
  }
#else
  if (p.o.variant == FO_VARIANT_PLAIN) factor(p, ln, alpha, negj, lu, w, alg_only);
  else if (p.o.variant == FO_VARIANT_COMPACT) {
    if (ln.L == 32) factor_compact<32>(p, ln, alpha, negj, lu, w, alg_only);
    else factor_compact<0>(p, ln, alpha, negj, lu, w, alg_only);
  } else {
    if (ln.L == 32) factor_stream<32>(p, ln, alpha, negj, lu, w, alg_only);
    else factor_stream<0>(p, ln, alpha, negj, lu, w, alg_only);
  }
#endif
}

__device__ __forceinline__ void solve_in_w(const SolveParams& p, const Lane& ln, const double* lu, double* w) {
  if (p.o.variant == FO_VARIANT_PLAIN) lu_solve(p, ln, lu, w);
  else if (ln.L == 32) lu_solve_pipelined<32>(p, ln, lu, w);
  else lu_solve_pipelined<0>(p, ln, lu, w);
}

// x = A^-1 b with the factors in lu (b and x per-lane vectors, may alias);
// alg_only: the factors are the projection's.
__device__ void solve_into(const SolveParams& p, const Lane& ln, const double* lu, double* w, const double* b,
                           double* x, bool alg_only = false) {
#ifdef FO_LINK_GENERATED
  // the generated solves work on the slot's solve vector (item xs), whose
  // offset they know, so every access is an immediate offset from one base
  double* base = const_cast<double*>(lu) - p.sl.lu * ln.L;
  double* xs = base + p.sl.xs * ln.L;
  if (b != xs) copy_items(ln, p.t.n, b, xs);
  if (alg_only) team_solve<true>(p, base + ln.lane);
  else team_solve<false>(p, base + ln.lane);
  if (x != xs) copy_items(ln, p.t.n, xs, x);
#else
  if (p.o.variant == FO_VARIANT_COMPACT) {
    lu_solve_compact(p, ln, lu, w, b, x);
    return;
  }
  const int L = ln.L, lane = ln.lane;
  for (int i = 0; i < p.t.n; ++i) WROW(i) = SCR(b, i);
  solve_in_w(p, ln, lu, w);
  for (int i = 0; i < p.t.n; ++i) SCR(x, i) = WROW(i);
#endif
}

// Sum over the block of one value per thread; every thread gets the same
// bits (xor butterfly, then the warp totals in warp order).
__device__ double block_sum(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  const int nw = blockDim.x >> 5;
  if (nw == 1) return v;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = red[0];
  for (int i = 1; i < nw; ++i) s += red[i];
  return s;
}

// A scalar that one warp of the team computes for all: f() by warp 0 of each
// block, handed on in shared memory (`slot`, one per use). Every warp takes the same
// decisions from it, and the FP64 units do its work once: with the
// controller's powers and divisions evaluated by all sixteen warps, an attempt
// of a 20-species mechanism took 142 us, with them done once 103 us.
template <class F>
__device__ __forceinline__ double team_once(double* slot, F f) {
  if (BLOCK_N == 1) return f();
  if (BLOCK_W == 0) {
    const double v = f();
    if (threadIdx.x == 0) *slot = v;
  }
  __syncthreads();
  return *slot;
}
// Slots of the reduction buffer (32 doubles, the first sixteen block_max's).
enum { kSlotError = 16, kSlotStep, kSlotAlpha, kSlotStart, kSlotPower, kSlotCoef = kSlotPower + 3 };

// err^(1/k) for the embedded order's k = 3.
__device__ __forceinline__ double error_root(double err) { return cbrt(err); }

// The filter's powers (err err_prev)^(-1/(b k)) and (H / h_prev)^(-1/b)
// (fastode/solvers.py:297-303), each by its own warp, or err^(1/k) alone. For
// the default b = 4 they are roots: about 2,500 cycles one after another where
// pow takes 12,000, with roundings of the same size.
__device__ __forceinline__ void team_powers(const DevOptions& o, double* red, bool filter, double err, double err_prev,
                                            double H, double h_prev, double (&v)[3]) {
  for (int q = BLOCK_W; q < 3; q += BLOCK_N) {
    if (filter != (q > 0)) continue;
    double r;
    if (q == 0) {
      r = error_root(err);
    } else {
      const double base = q == 1 ? __dmul_rn(err, err_prev) : __ddiv_rn(H, h_prev);
      if (o.b == 4.0) r = __ddiv_rn(1.0, sqrt(sqrt(q == 1 ? cbrt(base) : base)));
      else r = pow(base, q == 1 ? -1.0 / __dmul_rn(o.b, o.k_exp) : -1.0 / o.b);
    }
    if (BLOCK_N == 1) v[q] = r;
    else if (threadIdx.x == 0) red[kSlotPower + q] = r;
  }
  if (BLOCK_N == 1) return;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = red[kSlotPower + q];
}

// The scalars of an attempt of step H: returns alpha = 1 / (H gamma); a team
// divides it and the stages' c(r, s) / H side by side, one warp each.
__device__ __forceinline__ double attempt_scalars(const DevTableau& tb, double* red, double H) {
  if (BLOCK_N == 1) return 1.0 / __dmul_rn(H, tb.gamma);
  for (int q = BLOCK_W; q < 7; q += BLOCK_N) {
    const int r = q < 1 ? 1 : q < 3 ? 2 : 3;
    double v = 0.0;
    if (q == 6) v = 1.0 / __dmul_rn(H, tb.gamma);
    else if (r < tb.S) v = __ddiv_rn(tb.c[r][q - r * (r - 1) / 2], H);
    if (threadIdx.x == 0) red[q == 6 ? kSlotAlpha : kSlotCoef + q] = v;
  }
  __syncthreads();
  return red[kSlotAlpha];
}

// F (item f0; the generated form leaves it in ft) and the negated Jacobian at
// the step's start Y. `at_yr`: the last attempt left Y in item yr too (the
// generated form's evaluation point).
__device__ __forceinline__ void begin_step(const SolveParams& p, const Lane& ln, const double* Y, double* scr,
                                           bool at_yr) {
  const int L = ln.L;
#ifdef FO_LINK_GENERATED
  if (!at_yr) copy_items(ln, p.t.n, Y, scr + p.sl.yr * L);
  fo_gen_rhs(scr + ln.lane, TEAM_W, TEAM_N, p.o.gen_index);
  fo_gen_jac(scr + ln.lane, TEAM_W, TEAM_N, p.o.gen_index);
#else
  eval_rhs(p, ln, Y, scr + p.sl.r * L, scr + p.sl.f0 * L);
  eval_negjac(p, ln, Y, scr + p.sl.d * L, scr + p.sl.negj * L);
#endif
}

#ifdef FO_LINK_GENERATED
// numpy.maximum(|a|, |b|): for magnitudes the integer order is the numeric
// one, with NaN above everything, and the compare stays off the FP64 units.
__device__ __forceinline__ double max_magnitude(double a, double b) {
  const long long x = __double_as_longlong(fabs(a)), y = __double_as_longlong(fabs(b));
  return __longlong_as_double(x > y ? x : y);
}

// One attempt of the generated integrator (what `attempt` below does for the
// table-driven variants, the same operations in the same order), compiled for
// each tableau: its coefficients are immediates, products with zero and one
// are left out (which changes no value), and a stage's operands are loaded
// together. A stage's solution stays in the solve vector until the next loop
// over species reads it, which also stores it; the last one is stored only
// for the adjoint (U). `fresh`: F of the step's start is in item ft and is
// kept in f0 for further attempts. Y_new is left in item yr as well, the point
// of the next evaluation. With the loops driven by the tableau in memory these
// parts took 97,000 of an attempt's 195,000 cycles for a 20-species mechanism
// (team of 16).
template <int kTableau>
__device__ __noinline__ double attempt_generated(const SolveParams& p, const Lane& ln, double H, const double* Y_,
                                                 double* Ynew_, double* scr, double* red, double* U, bool fresh) {
  constexpr DevTableau tb = tableau_of(kTableau);
  constexpr int S = tb.S, kBatch = 4, kPartials = 16;
  const int n = p.t.n, lane = ln.lane, warp = TEAM_W, warps = TEAM_N, mech = p.o.gen_index;
  const bool dae = p.t.has_constraints != 0;
  double* const base = scr + lane;
  const double* const Y = Y_ + lane;
  double* const Ynew = Ynew_ + lane;
  double* const F0 = base + p.sl.f0 * 32;
  double* const Ft = base + p.sl.ft * 32;
  double* const Yr = base + p.sl.yr * 32;
  double* const xs = base + p.sl.xs * 32;
  double* const K = base + p.sl.k * 32;
  const double* const mass = p.t.mass;
  const int64_t kn = (int64_t)n * 32;
  bool anew = false;   // F was evaluated after the step's start
#pragma unroll
  for (int r = 0; r < S; ++r) {
    if (r > 0 && tb.new_forcing[r]) {
      for (int i0 = warp; i0 < n; i0 += kBatch * warps) {
        double y[kBatch], k[S][kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int i = i0 + b * warps;
          if (i >= n) continue;
          y[b] = Y[i * 32];
          k[r - 1][b] = xs[i * 32];
#pragma unroll
          for (int s = 0; s + 1 < r; ++s)
            if (tb.a[r][s] != 0.0) k[s][b] = K[s * kn + i * 32];
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int i = i0 + b * warps;
          if (i >= n) continue;
          double v = y[b];
#pragma unroll
          for (int s = 0; s < r; ++s)
            if (tb.a[r][s] != 0.0) v = __dadd_rn(v, tb.a[r][s] == 1.0 ? k[s][b] : __dmul_rn(tb.a[r][s], k[s][b]));
          K[(r - 1) * kn + i * 32] = k[r - 1][b];
          Yr[i * 32] = v;
          if (U != nullptr) U[r * kn + i * 32 + lane] = v;   // stage point kept for the adjoint
        }
      }
      fo_gen_rhs(base, warp, warps, mech);
      anew = true;
    }
    double coef[S];
#pragma unroll
    for (int s = 0; s < r; ++s)
      coef[s] = tb.c[r][s] == 0.0 ? 0.0
                : BLOCK_N > 1     ? red[kSlotCoef + r * (r - 1) / 2 + s]
                                  : __ddiv_rn(tb.c[r][s], H);
    const double* const f = anew || (r == 0 && fresh) ? Ft : F0;
    const bool keep = r == 0 && fresh;                    // F of the step's start into f0
    const bool move = r > 0 && !tb.new_forcing[r];        // the last solution into K
    for (int i0 = warp; i0 < n; i0 += kBatch * warps) {
      double v[kBatch], k[S][kBatch];
      long long m[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * warps;
        if (i >= n) continue;
        v[b] = f[i * 32];
#pragma unroll
        for (int s = 0; s < r; ++s)
          if (tb.c[r][s] != 0.0 || (move && s == r - 1))
            k[s][b] = move && s == r - 1 ? xs[i * 32] : K[s * kn + i * 32];
        if (r > 0 && dae) m[b] = __double_as_longlong(__ldg(mass + i));
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * warps;
        if (i >= n) continue;
        if (keep) F0[i * 32] = v[b];
        if (move) K[(r - 1) * kn + i * 32] = k[r - 1][b];
#pragma unroll
        for (int s = 0; s < r; ++s)
          if (tb.c[r][s] != 0.0) {
            double ks = k[s][b];
            if (dae && m[b] != 0x3ff0000000000000ll) ks = __dmul_rn(ks, __longlong_as_double(m[b]));
            v[b] = __dadd_rn(v[b], __dmul_rn(coef[s], ks));
          }
        xs[i * 32] = v[b];
      }
    }
    team_solve<false>(p, base);
  }
  // Y_new, E and the weighted sum of squares: min(n, 16) interleaved partial
  // sums (species s, s + 16, ...), added in order, whatever the team's size
  const int np = n < kPartials ? n : kPartials;
  const bool change = p.o.loop == FO_LOOP_RESTARTING && p.o.step_change_rows && dae;
  const double* const atol = p.atol;
  const int32_t* const perm = p.t.perm;
  const double rtol = p.rtol;
  // A team of several blocks leaves every species' square in ft first, each
  // by its own warp, for the partial sums to pick up: its DP work would
  // otherwise fall to the sixteen warps of one SM.
  const bool spread = warps > kPartials;
  const int stride = spread ? warps : np;
  for (int s0 = warp; s0 < (spread ? n : np); s0 += spread ? n : warps) {
    double acc = 0.0;
    for (int i0 = s0; i0 < n; i0 += kBatch * stride) {
      double y[kBatch], k[S][kBatch], tol[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * stride;
        if (i >= n) continue;
        tol[b] = __ldg(atol + __ldg(perm + i));
        y[b] = Y[i * 32];
#pragma unroll
        for (int r = 0; r < S; ++r)
          if (tb.m[r] != 0.0 || tb.e[r] != 0.0 || r == S - 1) k[r][b] = r == S - 1 ? xs[i * 32] : K[r * kn + i * 32];
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * stride;
        if (i >= n) continue;
        double yn = y[b], e = 0.0;
        bool first = true;
#pragma unroll
        for (int r = 0; r < S; ++r) {
          if (tb.m[r] != 0.0) yn = __dadd_rn(yn, tb.m[r] == 1.0 ? k[r][b] : __dmul_rn(tb.m[r], k[r][b]));
          if (tb.e[r] != 0.0) {
            const double term = tb.e[r] == 1.0 ? k[r][b] : __dmul_rn(tb.e[r], k[r][b]);
            e = first ? term : __dadd_rn(e, term);
            first = false;
          }
        }
        Ynew[i * 32] = yn;
        Yr[i * 32] = yn;
        if (U != nullptr) K[(S - 1) * kn + i * 32] = k[S - 1][b];
        // the restarting loop replaces the algebraic rows of the estimate by
        // the step change (fastode/solvers.py:238-239)
        if (change && __ldg(mass + i) == 0.0) e = __dsub_rn(yn, y[b]);
        const double q = __ddiv_rn(e, __dadd_rn(tol[b], __dmul_rn(rtol, max_magnitude(y[b], yn))));
        if (spread) Ft[i * 32] = __dmul_rn(q, q);
        else acc = __dadd_rn(acc, __dmul_rn(q, q));
      }
    }
    if (!spread) Ft[s0 * 32] = acc;
  }
  team_sync();
  if (spread) {
    // every block adds the partial sums up for itself, one per warp, in place
    // of the reduction buffer's other uses (32 lanes each)
    double* const sums = red + 32 + lane;
    const int w = BLOCK_W;
    if (w < np) {
      double acc = 0.0;
      for (int i = w; i < n; i += np) acc = __dadd_rn(acc, Ft[i * 32]);
      sums[w * 32] = acc;
    }
    __syncthreads();
    if (w != 0) return 0.0;
    double total = 0.0;
    for (int s0 = 0; s0 < np; ++s0) total = __dadd_rn(total, sums[s0 * 32]);
    return ln.active ? total : 0.0;
  }
  if (warp != 0) return 0.0;
  double part[kPartials], total = 0.0;
#pragma unroll
  for (int s0 = 0; s0 < kPartials; ++s0) part[s0] = s0 < np ? Ft[s0 * 32] : 0.0;
#pragma unroll
  for (int s0 = 0; s0 < kPartials; ++s0)
    if (s0 < np) total = __dadd_rn(total, part[s0]);
  return ln.active ? total : 0.0;
}

// A team returns the norm's sum in warp 0 of each block.
__device__ __forceinline__ double attempt(const SolveParams& p, const Lane& ln, double H, const double* Y, double* Ynew,
                                          double* scr, double*, double* red, long long& c_rhs, long long& c_solves,
                                          bool fresh, double* U = nullptr) {
  const bool ros3 = p.o.tableau == FO_TABLEAU_ROS3;
  c_rhs += ros3 ? 1 : 2;
  c_solves += ros3 ? 3 : 4;
  return ros3 ? attempt_generated<FO_TABLEAU_ROS3>(p, ln, H, Y, Ynew, scr, red, U, fresh)
              : attempt_generated<FO_TABLEAU_RODAS3>(p, ln, H, Y, Ynew, scr, red, U, fresh);
}
#else
// One attempt's stages (fastode/solvers.py:54-86), then Y_new, the error
// estimate and this lane's share of the error norm (fastode/solvers.py:37-43).
__device__ __noinline__ double attempt(const SolveParams& p, const Lane& ln, double H, const double* Y, double* Ynew,
                                       double* scr, double* w, double*, long long& c_rhs, long long& c_solves,
                                       bool, double* U = nullptr) {
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n;
  const DevTableau& tb = p.o.tab;
  const bool dae = p.t.has_constraints != 0;
  double* F0 = scr + p.sl.f0 * L;
  double* Ft = scr + p.sl.ft * L;
  double* Yr = scr + p.sl.yr * L;
  double* K = scr + p.sl.k * L;
  double* lu = scr + p.sl.lu * L;
  double* rr = scr + p.sl.r * L;
  const double* forcing = F0;
  constexpr int kBatch = 4;   // species of a warp whose loads are in flight together
  for (int r = 0; r < tb.S; ++r) {
    if (r > 0 && tb.new_forcing[r]) {
      for (int i0 = 0; i0 < n; i0 += kBatch) {
        double v[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (i0 + b < n) v[b] = SCR(Y, i0 + b);
        for (int s = 0; s < r; ++s)
          if (tb.a[r][s] != 0.0) {
            double ks[kBatch];
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
              if (i0 + b < n) ks[b] = SCR(K + (int64_t)s * n * L, i0 + b);
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
              if (i0 + b < n) v[b] = __dadd_rn(v[b], __dmul_rn(tb.a[r][s], ks[b]));
          }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int i = i0 + b;
          if (i >= n) continue;
          SCR(Yr, i) = v[b];
          if (U != nullptr) SCR(U + (int64_t)r * n * L, i) = v[b];   // stage point kept for the adjoint
        }
      }
      eval_rhs(p, ln, Yr, rr, Ft);
      ++c_rhs;
      forcing = Ft;
    }
    double* Kr = K + (int64_t)r * n * L;
    const bool in_place = solves_in_place(p);   // right-hand side in Kr, solved in place
    // the stage's c(r, s) / H once per stage rather than once per species
    // (the same quotients, so the same sums bit for bit)
    double coefs[4];
    for (int s = 0; s < r; ++s) coefs[s] = __ddiv_rn(tb.c[r][s], H);
    for (int i0 = 0; i0 < n; i0 += kBatch) {
      double v[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b)
        if (i0 + b < n) v[b] = SCR(forcing, i0 + b);
      for (int s = 0; s < r; ++s) {
        const double coef = coefs[s];
        if (coef == 0.0) continue;
        double ks[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int i = i0 + b;
          if (i >= n) continue;
          ks[b] = SCR(K + (int64_t)s * n * L, i);
          if (dae) ks[b] = __dmul_rn(ks[b], __ldg(p.t.mass + i));
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (i0 + b < n) v[b] = __dadd_rn(v[b], __dmul_rn(coef, ks[b]));
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b;
        if (i >= n) continue;
        if (in_place) SCR(Kr, i) = v[b];
        else WROW(i) = v[b];
      }
    }
    if (in_place) {
      solve_into(p, ln, lu, w, Kr, Kr);
    } else {
      solve_in_w(p, ln, lu, w);
      for (int i = 0; i < n; ++i) SCR(Kr, i) = WROW(i);
    }
    ++c_solves;
  }
  // Y_new, E and the weighted sum of squares: min(n, 16) interleaved partial
  // sums (species s, s + 16, ...), added in order, as the generated variant's
  // teams sum it
  constexpr int kPartials = 16;
  const int np = n < kPartials ? n : kPartials;
  for (int s0 = 0; s0 < np; ++s0) {
    double acc = 0.0;
    for (int i0 = s0; i0 < n; i0 += kBatch * np) {
      double yv[kBatch], yn[kBatch], e[kBatch], tol[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * np;
        if (i >= n) continue;
        yv[b] = yn[b] = SCR(Y, i);
        e[b] = 0.0;
        tol[b] = __ldg(p.atol + __ldg(p.t.perm + i));
      }
      for (int r = 0; r < tb.S; ++r) {
        double ks[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
          if (i0 + b * np < n) ks[b] = SCR(K + (int64_t)r * n * L, i0 + b * np);
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          if (i0 + b * np >= n) continue;
          if (tb.m[r] != 0.0) yn[b] = __dadd_rn(yn[b], __dmul_rn(tb.m[r], ks[b]));
          if (tb.e[r] != 0.0) e[b] = __dadd_rn(e[b], __dmul_rn(tb.e[r], ks[b]));
        }
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * np;
        if (i >= n) continue;
        SCR(Ynew, i) = yn[b];
        // the restarting loop replaces the algebraic rows of the estimate by
        // the step change (fastode/solvers.py:238-239)
        if (p.o.loop == FO_LOOP_RESTARTING && p.o.step_change_rows && dae && __ldg(p.t.mass + i) == 0.0)
          e[b] = __dsub_rn(yn[b], yv[b]);
        const double ymax = npmax(fabs(yv[b]), fabs(yn[b]));
        const double q = __ddiv_rn(e[b], __dadd_rn(tol[b], __dmul_rn(p.rtol, ymax)));
        acc = __dadd_rn(acc, __dmul_rn(q, q));
      }
    }
    SCR(Ft, s0) = acc;
  }
  double total = 0.0;
  for (int s0 = 0; s0 < np; ++s0) total = __dadd_rn(total, SCR(Ft, s0));
  return ln.active ? total : 0.0;
}
#endif

__device__ void trace_record(const SolveParams& p, int g, int& nrec, double t, double H, double err, double outcome) {
  if (p.trace == nullptr || !team_leader()) {
    ++nrec;
    return;
  }
  if (nrec < p.trace_cap) {
    double* rec = p.trace + ((int64_t)g * p.trace_cap + nrec) * 4;
    rec[0] = t;
    rec[1] = H;
    rec[2] = err;
    rec[3] = outcome;
  }
  ++nrec;
}

// One double per block of a cluster, of each block's v, for every block: in
// the slot's partial derivatives and rates (R items or more, so R is at least
// kMaxCluster wherever clusters run), which no evaluation uses here.
__device__ __forceinline__ void cluster_gather(const SolveParams& p, double v, double (&all)[kMaxCluster]) {
#ifdef FO_LINK_GENERATED
  const int blocks = cluster_blocks();
  double* const at = p.scratch + (int64_t)(blockIdx.x / blocks) * p.slot_doubles + p.sl.d * 32;
  if (threadIdx.x == 0 && BLOCK_W == 0) at[cluster_rank() * 32] = v;
  team_sync();
#pragma unroll
  for (int b = 0; b < kMaxCluster; ++b) all[b] = b < blocks ? at[b * 32] : v;
  team_sync();
#endif
}

// Team-wide max with NaN propagation (numpy max) and team-wide AND.
__device__ double block_max(const SolveParams& p, double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v = npmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  const int nw = (blockDim.x >> 5) * BLOCK_N;
  if (nw == 1) return v;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[(threadIdx.x >> 5) + BLOCK_W] = v;
  __syncthreads();
  double s = red[0];
  for (int i = 1; i < nw; ++i) s = npmax(s, red[i]);
  if (cluster_team()) {
    double all[kMaxCluster];
    cluster_gather(p, s, all);
#pragma unroll
    for (int b = 0; b < kMaxCluster; ++b) s = npmax(s, all[b]);
  }
  return s;
}

__device__ bool block_all(const SolveParams& p, bool v) {
  bool all_true = __syncthreads_and(v ? 1 : 0) != 0;
  if (cluster_team()) {
    double all[kMaxCluster];
    cluster_gather(p, all_true ? 1.0 : 0.0, all);
#pragma unroll
    for (int b = 0; b < kMaxCluster; ++b) all_true = all_true && all[b] != 0.0;
  }
  return all_true;
}

struct ProjectionCounts {
  long long rhs = 0, jac = 0, lu = 0, solves = 0, passes = 0, trials = 0;
};

// All algebraic entries of A (a per-lane vector) finite, over the group.
__device__ bool alg_finite(const SolveParams& p, const Lane& ln, const double* A) {
  const int L = ln.L, lane = ln.lane;
  bool ok = true;
  if (ln.active)
    for (int i = TEAM_W; i < p.t.n; i += TEAM_N)
      if (__ldg(p.t.mass + i) == 0.0 && !isfinite(SCR(A, i))) ok = false;
  return block_all(p, ok);
}

// max over the group's algebraic entries of |A|
__device__ double alg_absmax(const SolveParams& p, const Lane& ln, const double* A, double* red) {
  const int L = ln.L, lane = ln.lane;
  double m = 0.0;
  if (ln.active)
    for (int i = TEAM_W; i < p.t.n; i += TEAM_N)
      if (__ldg(p.t.mass + i) == 0.0) m = npmax(m, fabs(SCR(A, i)));
  return block_max(p, m, red);
}

// The weighted Newton correction of fastode/solvers.py:119-124:
// max over algebraic entries of |d| / (atol + rtol max(|z|, |z + d|)), with
// 0 where d = 0 and the scale vanishes, inf where only the scale vanishes.
__device__ double weighted(const SolveParams& p, const Lane& ln, const double* Z, const double* D, double* red) {
  const int L = ln.L, lane = ln.lane;
  double m = 0.0;
  if (ln.active)
    for (int i = TEAM_W; i < p.t.n; i += TEAM_N) {
      if (__ldg(p.t.mass + i) != 0.0) continue;
      const double z = SCR(Z, i), d = SCR(D, i);
      const double scale =
          __dadd_rn(__ldg(p.atol + __ldg(p.t.perm + i)), __dmul_rn(p.rtol, npmax(fabs(z), fabs(__dadd_rn(z, d)))));
      double q;
      if (scale > 0.0) q = __ddiv_rn(fabs(d), scale);
      else if (scale != scale) q = scale;
      else q = (d == 0.0) ? 0.0 : CUDART_INF;
      m = npmax(m, q);
    }
  return block_max(p, m, red);
}

// G = F(Z) with the differential rows zeroed (fastode/solvers.py:110-114).
__device__ void alg_residual(const SolveParams& p, const Lane& ln, const double* Z, double* rr, double* G) {
  const int L = ln.L, lane = ln.lane;
  eval_rhs(p, ln, Z, rr, G);
  for (int i = TEAM_W; i < p.t.n; i += TEAM_N)
    if (__ldg(p.t.mass + i) != 0.0) SCR(G, i) = 0.0;
}


// Consistent initialization of the algebraic species, fastode/solvers.py:100-178:
// damped Newton with the algebraic-rows-only matrix (alpha = 1), accepted on
// the weighted correction, with backtracking line search. Returns true on
// convergence; on failure Y is restored to its value on entry.
// Every accepted update (Y += step * delta on the algebraic rows) is traced
// as (0, step, q, 2), so that the adjoint can replay the same updates.
__device__ __noinline__ bool project(const SolveParams& p, const Lane& ln, double* Y, double* scr, double* w, double* red,
                        ProjectionCounts& pc, int g, int& nrec) {
  const int L = ln.L, lane = ln.lane;
  const int n = p.t.n;
  double* G = scr + p.sl.f0 * L;
  double* cand = scr + p.sl.yr * L;
  double* orig = scr + p.sl.ynew * L;
  double* delta = scr + p.sl.k * L;
  double* trial = scr + (p.sl.k + n) * L;
  double* Gc = scr + p.sl.ft * L;
  double* rr = scr + p.sl.r * L;
  double* negj = scr + p.sl.negj * L;
  double* dd = scr + p.sl.d * L;
  double* lu = scr + p.sl.lu * L;
  const int max_updates = 10, max_backtracks = 24;
  const double tol = 0.1, factor_bt = 0.5, sigma = 1.0e-4;
  bool have_orig = false;
  for (int update = 0; update <= max_updates; ++update) {
    alg_residual(p, ln, Y, rr, G);
    ++pc.rhs;
    if (!alg_finite(p, ln, G)) break;
    ++pc.passes;
    if (alg_absmax(p, ln, G, red) == 0.0) return true;
    eval_negjac(p, ln, Y, dd, negj);
    ++pc.jac;
    factor_any(p, ln, 1.0, negj, lu, w, true);
    ++pc.lu;
    solve_into(p, ln, lu, w, G, delta, true);
    ++pc.solves;
    if (!alg_finite(p, ln, delta)) break;
    const double q = weighted(p, ln, Y, delta, red);
    if (q <= tol) return true;
    if (update == max_updates) break;
    if (!have_orig) {
      for (int i = TEAM_W; i < n; i += TEAM_N) SCR(orig, i) = SCR(Y, i);
      have_orig = true;
    }
    double step = 1.0, step_used = 0.0;
    bool accepted = false;
    for (int bt = 0; bt <= max_backtracks; ++bt) {
      for (int i = TEAM_W; i < n; i += TEAM_N) {
        double v = SCR(Y, i);
        if (__ldg(p.t.mass + i) == 0.0) v = __dadd_rn(v, __dmul_rn(step, SCR(delta, i)));
        SCR(cand, i) = v;
      }
      step_used = step;
      step = __dmul_rn(step, factor_bt);
      if (!alg_finite(p, ln, cand)) continue;
      alg_residual(p, ln, cand, rr, Gc);
      ++pc.trials;
      ++pc.rhs;
      if (!alg_finite(p, ln, Gc)) continue;
      if (alg_absmax(p, ln, Gc, red) == 0.0) {
        accepted = true;
        break;
      }
      solve_into(p, ln, lu, w, Gc, trial, true);
      ++pc.solves;
      if (!alg_finite(p, ln, trial)) continue;
      const double qt = weighted(p, ln, cand, trial, red);
      if (qt <= tol || qt < __dmul_rn(__dsub_rn(1.0, __dmul_rn(sigma, step_used)), q)) {
        accepted = true;
        break;
      }
    }
    if (!accepted) break;
    trace_record(p, g, nrec, 0.0, step_used, q, 2.0);
    for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Y, i) = SCR(cand, i);
  }
  if (have_orig)
    for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Y, i) = SCR(orig, i);
  return false;
}

// One group over one interval: fastode/solvers.py:305-415 statement by statement.
// The baseline restarting loop, fastode/solvers.py:205-267 statement by
// statement: a restart at 1e-6 of the interval, the elementary controller,
// no carried memory, "too many steps" past max_steps attempts.
__device__ __noinline__ void solve_group_restarting(const SolveParams& p, int g, double* scr, double* w,
                                                    double* red) {
  const int L = blockDim.x, lane = threadIdx.x;
  const int n = p.t.n;
  const int64_t c0 = p.group_offsets[g], C = p.group_offsets[g + 1] - c0;
  Lane ln;
  ln.lane = lane;
  ln.L = L;
  ln.active = lane < C;
  ln.cell = c0 + (ln.active ? lane : (C - 1));
  const DevOptions& o = p.o;
  const double dt = p.dt;
  long long c_steps = 0, c_acc = 0, c_rej = 0, c_rhs = 0, c_jac = 0, c_lu = 0, c_solves = 0;
  int nrec = 0;
  double* Y = scr + p.sl.y * L;
  double* Ynew = scr + p.sl.ynew * L;
  double* negj = scr + p.sl.negj * L;
  double* lu = scr + p.sl.lu * L;
  load_rate_constants(p, ln, scr);
  for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Y, i) = p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss];
  const double rounding = 2.220446049250313e-16;
  const double h_min = __dmul_rn(1.0e-15, dt);
  const double h_max = dt;
  double H = pymin(pymax(h_min, __dmul_rn(1.0e-6, dt)), h_max);
  const double nsize = (double)(C * n);
  int status = -1;
  ProjectionCounts pc;
  if (p.t.has_constraints && !project(p, ln, Y, scr, w, red, pc, g, nrec)) status = FO_STATUS_PROJECTION_FAILED;
  c_rhs += pc.rhs;
  c_jac += pc.jac;
  c_lu += pc.lu;
  c_solves += pc.solves;
  double t = 0.0;
  bool reject_last = false, reject_more = false, at_yr = false;
  int nsteps = 0;
  while (status < 0 && __dadd_rn(__dsub_rn(t, dt), rounding) <= 0.0) {
    if (nsteps > o.max_steps) {
      status = FO_STATUS_TOO_MANY_STEPS;
      break;
    }
    if (__dadd_rn(t, __dmul_rn(0.1, H)) == t || H <= pymin(rounding, h_min)) {
      status = FO_STATUS_STEP_TOO_SMALL;
      break;
    }
    H = pymin(H, fabs(__dsub_rn(dt, t)));
    begin_step(p, ln, Y, scr, at_yr);
    at_yr = true;
    ++c_rhs;
    ++c_jac;
    bool fresh = true;
    bool accepted = false;
    while (!accepted) {
      const double alpha = attempt_scalars(o.tab, red, H);
      factor_any(p, ln, alpha, negj, lu, w, false);
      ++c_lu;
      const double part = attempt(p, ln, H, Y, Ynew, scr, w, red, c_rhs, c_solves, fresh);
      fresh = false;
      const double err = team_once(red + kSlotError, [&] {
        const double e = sqrt(__ddiv_rn(block_sum(part, red), nsize));
        return isnan(e) ? e : pymax(e, 1.0e-10);
      });
      ++nsteps;
      ++c_steps;
      if (isnan(err) || isinf(err)) {
        trace_record(p, g, nrec, t, H, err, -1.0);
        status = FO_STATUS_NAN_OR_INF;
        break;
      }
      double Hnew = team_once(red + kSlotStep, [&] {
        return __dmul_rn(H, pymin(6.0, pymax(0.2, __ddiv_rn(0.9, error_root(err)))));
      });
      if (err < 1.0 || H < h_min) {
        trace_record(p, g, nrec, t, H, err, 1.0);
        ++c_acc;
        t = __dadd_rn(t, H);
        double* tmp = Y;
        Y = Ynew;
        Ynew = tmp;
        Hnew = pymax(h_min, pymin(Hnew, h_max));
        if (reject_last) Hnew = pymin(Hnew, H);
        reject_last = reject_more = false;
        H = Hnew;
        accepted = true;
      } else {
        trace_record(p, g, nrec, t, H, err, 0.0);
        if (reject_more) Hnew = __dmul_rn(H, 0.1);
        reject_more = reject_last;
        reject_last = true;
        H = Hnew;
        ++c_rej;
      }
    }
  }
  if (status < 0) status = FO_STATUS_CONVERGED;
  const bool clamp = status != FO_STATUS_PROJECTION_FAILED;
  if (ln.active)
    for (int i = TEAM_W; i < n; i += TEAM_N) {
      double y = SCR(Y, i);
      if (clamp && (!p.t.has_constraints || __ldg(p.t.mass + i) == 1.0)) y = clamp0(y);
      p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss] = y;
    }
  if (team_leader()) {
    long long* cn = p.counts + (int64_t)g * FO_NUM_COUNTS;
    cn[0] += c_steps;
    cn[1] += c_acc;
    cn[2] += c_rej;
    cn[3] += c_rhs;
    cn[4] += c_jac;
    cn[5] += c_lu;
    cn[6] += c_solves;
    cn[10] += pc.passes;
    cn[11] += pc.trials;
    cn[12] += 1;
    p.status[g] = status;
    if (p.trace_len) p.trace_len[g] = nrec;
  }
}

// The baseline backward Euler, fastode/solvers.py:439-491 statement by
// statement: every Newton iteration evaluates F and J at the iterate, factors
// M/H - J and solves for the update; the iterate is clamped at zero after
// each update. From the second iteration on, the step has converged when
// every update of the group is finite and within max(small, atol, rtol |Y|).
// A failed step restarts from the last accepted state with H cut by the next
// reduction; past the last reduction the unconverged iterate is accepted and
// the call ends. Two converged steps in a row double H.
__device__ __noinline__ void solve_group_backward_euler(const SolveParams& p, int g, double* scr, double* w,
                                                        double* red) {
  const int L = blockDim.x, lane = threadIdx.x;
  const int n = p.t.n;
  const int64_t c0 = p.group_offsets[g], C = p.group_offsets[g + 1] - c0;
  Lane ln;
  ln.lane = lane;
  ln.L = L;
  ln.active = lane < C;
  ln.cell = c0 + (ln.active ? lane : (C - 1));
  const DevOptions& o = p.o;
  const double dt = p.dt;
  long long c_steps = 0, c_acc = 0, c_rej = 0, c_rhs = 0, c_jac = 0, c_lu = 0, c_solves = 0;
  long long c_newton = 0, c_fail = 0, c_unconv = 0;
  double* Yn = scr + p.sl.y * L;
  double* Yn1 = scr + p.sl.ynew * L;
  double* F = scr + p.sl.f0 * L;
  double* negj = scr + p.sl.negj * L;
  double* dd = scr + p.sl.d * L;
  double* rr = scr + p.sl.r * L;
  double* lu = scr + p.sl.lu * L;
  const bool in_place = solves_in_place(p);   // Newton update solved in place in F
  load_rate_constants(p, ln, scr);
  for (int i = TEAM_W; i < n; i += TEAM_N) {
    const double v = p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss];
    SCR(Yn, i) = v;
    SCR(Yn1, i) = v;
  }
  double H = dt, t = 0.0;
  int n_success = 0, n_fail = 0;
  int status = FO_STATUS_CONVERGED;
  while (t < dt) {
    if (c_steps >= o.max_steps) {   // a guard of this build: the reference's loop has no budget
      status = FO_STATUS_TOO_MANY_STEPS;
      break;
    }
    bool ok = false;
    int iterations = 0;
    for (;;) {
      ++c_newton;
      eval_rhs(p, ln, Yn1, rr, F);
      ++c_rhs;
      eval_negjac(p, ln, Yn1, dd, negj);
      ++c_jac;
      factor_any(p, ln, 1.0 / H, negj, lu, w, false);
      ++c_lu;
      for (int i = TEAM_W; i < n; i += TEAM_N) {
        const double v = __dsub_rn(SCR(F, i), __ddiv_rn(__dsub_rn(SCR(Yn1, i), SCR(Yn, i)), H));
        if (in_place) SCR(F, i) = v;
        else WROW(i) = v;
      }
      if (in_place) solve_into(p, ln, lu, w, F, F);
      else solve_in_w(p, ln, lu, w);
      ++c_solves;
      ++iterations;
      bool conv = true;
      for (int i = TEAM_W; i < n; i += TEAM_N) {
        const double d = in_place ? SCR(F, i) : WROW(i);
        const double y = clamp0(__dadd_rn(SCR(Yn1, i), d));
        SCR(Yn1, i) = y;
        if (iterations > 1) {
          const double bound = npmax(npmax(o.small, __ldg(p.atol + __ldg(p.t.perm + i))), __dmul_rn(p.rtol, fabs(y)));
          conv = conv && isfinite(d) && fabs(d) <= bound;
        }
      }
      if (iterations > 1) ok = block_all(p, !ln.active || conv);
      if (ok || iterations >= o.max_iterations) break;
    }
    ++c_steps;
    if (!ok) {
      ++c_rej;
      ++c_fail;
      n_success = 0;
      if (n_fail >= o.nreductions) {
        t = __dadd_rn(t, H);
        ++c_unconv;
        status = FO_STATUS_ACCEPTED_UNCONVERGED;
        bool finite = true;
        for (int i = TEAM_W; i < n; i += TEAM_N) finite = finite && isfinite(SCR(Yn1, i));
        if (!block_all(p, !ln.active || finite)) status = FO_STATUS_NAN_OR_INF;
        break;
      }
      for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Yn1, i) = SCR(Yn, i);
      H = __dmul_rn(H, o.reductions[n_fail]);
      ++n_fail;
    } else {
      ++c_acc;
      t = __dadd_rn(t, H);
      for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Yn, i) = SCR(Yn1, i);
      ++n_success;
      if (n_success >= 2) {
        n_success = 0;
        H = __dmul_rn(H, 2.0);
      }
    }
    H = pymin(H, __dsub_rn(dt, t));
  }
  if (ln.active)
    for (int i = TEAM_W; i < n; i += TEAM_N) {
      double y = SCR(Yn1, i);
      if (!p.t.has_constraints || __ldg(p.t.mass + i) == 1.0) y = clamp0(y);
      p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss] = y;
    }
  if (team_leader()) {
    long long* cn = p.counts + (int64_t)g * FO_NUM_COUNTS;
    cn[0] += c_steps;
    cn[1] += c_acc;
    cn[2] += c_rej;
    cn[3] += c_rhs;
    cn[4] += c_jac;
    cn[5] += c_lu;
    cn[6] += c_solves;
    cn[7] += c_newton;
    cn[8] += c_fail;
    cn[9] += c_unconv;
    cn[12] += 1;
    p.status[g] = status;
    if (p.trace_len) p.trace_len[g] = 0;
  }
}

// Lockstep rounds. The blocks of an SM make their attempts in rounds: each
// block makes one attempt (of a small mechanism in a several-mechanism launch as
// many as cost about one of the largest, of one group after another), then
// waits for the SM's others. The straight-line code is megabytes, so warps that
// drift apart each stream their own instructions and thrash the SM's
// instruction cache; rounds keep them at the same place. The blocks of a round
// also meet before the solves: the scheduler favours an SM's oldest warps, so
// groups leave the factorization, which fills the FP64 units, one after
// another, and the youngest would make its solves, which wait on memory and on
// one another, with the SM to itself (one settled interval of 65,536 cells of
// the 210/500 mechanism 120 ms without the second meeting and 110 with it).
//
// An SM's state is one word: the blocks that take part (bits 0-7), those that
// have arrived at the meeting (8-15) and the meetings so far (16-31), even
// before a round's solves. A block joins when it starts and leaves when it has
// no group left, so nothing has to be resident but the blocks that wait, and a
// launch of any size can run in rounds on the plain launch's even placement.
// With one barrier over the whole grid every SM waited for the fullest, and the
// cooperative launch that it needs filled one SM after another (65,536 cells
// of 210/500 on 128 of 152 SMs). Grid-wide rounds and an SM's, ms: one cold
// interval of 210/500, 9,600 cells 139 and 119, 13,000 185 and 163, 16,384 226
// and 206, 65,536 756 and 716; three mechanisms, 196,608 cells, settled (where
// grid-wide rounds lost to none) 136 and 112, cold 1019 and 856.
//
// The rounds only order time: no group reads another's data, so results are
// those of the unsynchronized launch bit for bit. A wait is bounded
// (kRoundSpinLimit polls about 1 us apart, some 30 s); a block that gives up
// leaves the rounds and runs on without them.
constexpr int kRoundSpinLimit = 30000000;
constexpr unsigned int kRoundMember = 1u, kRoundArrival = 1u << 8, kRoundMeeting = 1u << 16;

// Adds `change` to an SM's state and holds the meeting if that completes it;
// returns the state before.
__device__ __forceinline__ unsigned int round_update(unsigned int* w, unsigned int change) {
  unsigned int old = *reinterpret_cast<volatile unsigned int*>(w);
  for (;;) {
    unsigned int s = old + change;
    if ((s & 0xffu) != 0u && (s >> 8 & 0xffu) == (s & 0xffu)) s = (s & 0xffff00ffu) + kRoundMeeting;
    const unsigned int seen = atomicCAS(w, old, s);
    if (seen == old) return old;
    old = seen;
  }
}

// Where a block is in its round: its SM's state (null: no rounds), the units
// done, and whether it has met the others before the solves. It carries over
// from group to group.
struct RoundPace {
  unsigned int* state = nullptr;
  int done = 0;
  bool met = false;
};

// Waits for the SM's other blocks. Every thread of the block calls it.
__device__ void round_meet(RoundPace& pace) {
  __shared__ int held;
  __syncthreads();
  if (team_leader()) {
    const volatile unsigned int* state = pace.state;
    const unsigned int meeting = round_update(pace.state, kRoundArrival) >> 16;
    for (int spins = 0; *state >> 16 == meeting && spins < kRoundSpinLimit; ++spins) __nanosleep(1000);
    held = 1;
    unsigned int s = *state;
    while (s >> 16 == meeting) {   // given up: neither a member nor arrived any more
      unsigned int left = s - kRoundMember - kRoundArrival;
      if ((left & 0xffu) != 0u && (left >> 8 & 0xffu) == (left & 0xffu)) left = (left & 0xffff00ffu) + kRoundMeeting;
      const unsigned int seen = atomicCAS(pace.state, s, left);
      held = seen == s ? 0 : 1;
      if (seen == s) break;
      s = seen;
    }
  }
  __syncthreads();
  if (!held) pace.state = nullptr;
}

// The block joins its SM's rounds (`words` null: none), between two rounds:
// where the others are at their solves it waits for them to finish.
__device__ void rounds_join(unsigned int* words, RoundPace& pace) {
  __shared__ int at, wait;
  if (words == nullptr) return;
  if (team_leader()) {
    unsigned int sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    at = (int)(sm % kRoundStates) * kRoundStride;
    unsigned int* w = words + at;
    unsigned int old = *reinterpret_cast<volatile unsigned int*>(w);
    for (;;) {
      const bool first = (old & 0xffu) == 0u, solves = (old >> 16 & 1u) != 0u;
      const unsigned int s = old + kRoundMember + (first && solves ? kRoundMeeting : 0u);
      const unsigned int seen = atomicCAS(w, old, s);
      if (seen == old) {
        wait = !first && solves;
        break;
      }
      old = seen;
    }
  }
  __syncthreads();
  pace.state = words + at;
  if (wait) round_meet(pace);
}

__device__ __forceinline__ void rounds_leave(RoundPace& pace) {
  if (pace.state != nullptr && team_leader()) round_update(pace.state, 0u - kRoundMember);
}

// The parameters of batch b of a several-mechanism launch, copied from the
// batch table in global memory into the block's shared copy when the block
// moves to another batch, so that the integrator's parameter reads do not
// compete with the factorization's operand stream for L1. Every thread of
// the block calls this.
__device__ __forceinline__ void load_batch_params(const SolveParams* __restrict__ batches, int b, int& current,
                                                  SolveParams& shared) {
  static_assert(sizeof(SolveParams) % sizeof(long long) == 0, "SolveParams copies as 8-byte words");
  if (b == current) return;
  __syncthreads();
  const long long* src = reinterpret_cast<const long long*>(batches + b);
  long long* dst = reinterpret_cast<long long*>(&shared);
  for (int i = threadIdx.x; TEAM_W == 0 && i < (int)(sizeof(SolveParams) / sizeof(long long)); i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  current = b;
}

// The block has done `units` more of its round.
__device__ __forceinline__ void round_advance(RoundPace& pace, int units) {
  pace.done += units;
  if (!pace.met && pace.done >= kRoundSolves) {
    pace.met = true;
    round_meet(pace);
    if (pace.state == nullptr) return;
  }
  if (pace.met && pace.done >= kRoundUnits) {
    pace.met = false;
    pace.done -= kRoundUnits;
    round_meet(pace);
  }
}

__device__ void solve_group_algorithm(const SolveParams& p, int g, double* scr, double* w, double* red,
                                      RoundPace& pace);

__device__ void solve_group(const SolveParams& p, int g, double* scr, double* w, double* red, RoundPace& pace) {
  if (p.o.loop == FO_LOOP_RESTARTING) solve_group_restarting(p, g, scr, w, red);
  else if (p.o.loop == FO_LOOP_BACKWARD_EULER) solve_group_backward_euler(p, g, scr, w, red);
  else solve_group_algorithm(p, g, scr, w, red, pace);
}

__device__ void solve_group_algorithm(const SolveParams& p, int g, double* scr, double* w, double* red,
                                      RoundPace& pace) {
  const int L = blockDim.x, lane = threadIdx.x;
  const int n = p.t.n;
  const int64_t c0 = p.group_offsets[g], c1 = p.group_offsets[g + 1];
  const int64_t C = c1 - c0;
  Lane ln;
  ln.lane = lane;
  ln.L = L;
  ln.active = lane < C;
  ln.cell = c0 + (ln.active ? lane : (C - 1));
  const DevOptions& o = p.o;
  const double dt = p.dt;

  long long c_steps = 0, c_acc = 0, c_rej = 0, c_rhs = 0, c_jac = 0, c_lu = 0, c_solves = 0;
  int nrec = 0;

  double* Y = scr + p.sl.y * L;
  double* Ynew = scr + p.sl.ynew * L;
  double* negj = scr + p.sl.negj * L;
  double* lu = scr + p.sl.lu * L;

  load_rate_constants(p, ln, scr);
  for (int i = TEAM_W; i < n; i += TEAM_N) SCR(Y, i) = p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss];

  double* mem = p.memory + (int64_t)g * 3;
  double h_next = mem[0], err_prev = mem[1], h_prev = mem[2];
  if (cluster_team()) team_sync();   // no block writes the memory before all have read it
  if (!(o.carry && o.carry_memory)) err_prev = h_prev = 0.0;
  const double h_min = __dmul_rn(1.0e-15, dt);
  const double h_max = dt;
  double H = (o.carry && h_next > 0.0) ? h_next : __dmul_rn(1.0e-6, dt);
  H = pymin(pymax(h_min, H), h_max);
  H = team_once(red + kSlotStart, [&] { return o.quantize ? quantize_step(H, dt) : H; });
  double proposed = H;
  const double up = 1.0 + 1.0e-8, down = 1.0 - 1.0e-8;
  const double rounding = 2.220446049250313e-16;

  double t = 0.0;
  bool reject_last = false, reject_more = false, at_yr = false;
  int nsteps = 0;
  int status = -1;  // running
  const double nsize = (double)(C * n);
  ProjectionCounts pc;
  if (p.t.has_constraints && !project(p, ln, Y, scr, w, red, pc, g, nrec)) {
    status = FO_STATUS_PROJECTION_FAILED;   // Y restored, no step taken
    proposed = h_next;                      // the carried proposal is left as it was
  }
  c_rhs += pc.rhs;
  c_jac += pc.jac;
  c_lu += pc.lu;
  c_solves += pc.solves;
  while (status < 0 && __dadd_rn(__dsub_rn(t, dt), rounding) <= 0.0) {
    if (nsteps >= o.max_steps) {
      status = FO_STATUS_TOO_MANY_STEPS;
      break;
    }
    if (__dadd_rn(t, __dmul_rn(0.1, H)) == t || H < h_min) {
      status = FO_STATUS_STEP_TOO_SMALL;
      break;
    }
    bool last = __dsub_rn(dt, t) <= __dmul_rn(H, up);
    bool shortened = last && __dsub_rn(dt, t) < __dmul_rn(H, down);
    double H_ctrl = H;
    if (last) H = __dsub_rn(dt, t);
    begin_step(p, ln, Y, scr, at_yr);
    at_yr = true;
    ++c_rhs;
    ++c_jac;
    bool fresh = true;
    bool accepted = false;
    while (!accepted) {
      if (nsteps >= o.max_steps) {
        status = FO_STATUS_TOO_MANY_STEPS;
        break;
      }
      if (H < h_min || __dadd_rn(t, __dmul_rn(0.1, H)) == t) {
        status = FO_STATUS_STEP_TOO_SMALL;
        break;
      }
      const double alpha = attempt_scalars(o.tab, red, H);
      factor_any(p, ln, alpha, negj, lu, w, false);
      ++c_lu;
      const int to_solves = p.round_cost * kRoundSolves / kRoundUnits;
      if (pace.state != nullptr) round_advance(pace, to_solves);
      const double part = attempt(p, ln, H, Y, Ynew, scr, w, red, c_rhs, c_solves, fresh);
      fresh = false;
      const double err = team_once(red + kSlotError, [&] {
        const double e = sqrt(__ddiv_rn(block_sum(part, red), nsize));
        return isnan(e) ? e : pymax(e, 1.0e-10);
      });
      ++nsteps;
      ++c_steps;
      if (isnan(err) || isinf(err)) {
        trace_record(p, g, nrec, t, H, err, -1.0);
        status = FO_STATUS_NAN_OR_INF;
        // the round ends here too: half of one carried to the block's next
        // group would put that one's solves among the others' factorizations
        if (pace.state != nullptr) round_advance(pace, p.round_cost - to_solves);
        break;
      }
      if (err < 1.0 && shortened) {
        trace_record(p, g, nrec, t, H, err, 1.0);
        ++c_acc;
        t = dt;
        double* tmp = Y; Y = Ynew; Ynew = tmp;
        proposed = H_ctrl;
        accepted = true;
      } else if (err < 1.0) {
        trace_record(p, g, nrec, t, H, err, 1.0);
        // fastode/solvers.py:297-303
        const bool filter = o.controller == FO_CONTROLLER_H211B && err_prev > 0.0 && h_prev > 0.0;
        double pw[3];
        team_powers(o, red, filter, err, err_prev, H, h_prev, pw);
        ++c_acc;
        t = last ? dt : __dadd_rn(t, H);
        double* tmp = Y; Y = Ynew; Ynew = tmp;
        err_prev = err;
        h_prev = H;
        const double Hnew = team_once(red + kSlotStep, [&] {
          double fac = filter ? __dmul_rn(__dmul_rn(o.safety, pw[1]), pw[2]) : __ddiv_rn(o.safety, pw[0]);
          fac = pymin(o.fac_max, pymax(o.fac_min, fac));
          double h = __dmul_rn(H, fac);
          if (reject_last) h = pymin(h, H);
          h = pymax(h_min, pymin(h, h_max));
          return o.quantize ? quantize_step(h, dt) : h;
        });
        reject_last = reject_more = false;
        proposed = Hnew;
        H = Hnew;
        accepted = true;
      } else {
        trace_record(p, g, nrec, t, H, err, 0.0);
        const double Hnew = team_once(red + kSlotStep, [&] {
          double h = __dmul_rn(H, pymax(o.fac_min, __ddiv_rn(o.safety, error_root(err))));
          if (reject_more) h = __dmul_rn(H, 0.1);
          return o.quantize ? quantize_step(h, dt) : h;
        });
        reject_more = reject_last;
        reject_last = true;
        H = Hnew;
        last = __dsub_rn(dt, t) <= __dmul_rn(H, up);
        shortened = last && __dsub_rn(dt, t) < __dmul_rn(H, down);
        H_ctrl = H;
        if (last) H = __dsub_rn(dt, t);
        ++c_rej;
      }
      if (pace.state != nullptr) round_advance(pace, p.round_cost - to_solves);
    }
  }
  if (status < 0) status = FO_STATUS_CONVERGED;

  // clamp (fastode/solvers.py:89-97) and write back; a failed projection
  // returns the restored state unclamped (fastode/solvers.py:323-325)
  const bool clamp = status != FO_STATUS_PROJECTION_FAILED;
  if (ln.active) {
    for (int i = TEAM_W; i < n; i += TEAM_N) {
      double y = SCR(Y, i);
      if (clamp && (!p.t.has_constraints || __ldg(p.t.mass + i) == 1.0)) y = clamp0(y);
      p.Y[ln.cell * p.ycs + (int64_t)__ldg(p.t.perm + i) * p.yss] = y;
    }
  }
  if (team_leader()) {
    mem[0] = proposed;
    mem[1] = err_prev;
    mem[2] = h_prev;
    long long* cn = p.counts + (int64_t)g * FO_NUM_COUNTS;
    cn[0] += c_steps;
    cn[1] += c_acc;
    cn[2] += c_rej;
    cn[3] += c_rhs;
    cn[4] += c_jac;
    cn[5] += c_lu;
    cn[6] += c_solves;
    cn[10] += pc.passes;
    cn[11] += pc.trials;
    cn[12] += 1;
    p.status[g] = status;
    if (p.trace_len) p.trace_len[g] = nrec;
  }
}

}  // namespace
}  // namespace fo

