// The integrator kernels of the generated variant (FO_VARIANT_GENERATED).
//
// This translation unit is compiled once, at build time, as relocatable
// device code (nvcc -rdc=true -cubin); it calls the phases that a plan
// generates for its own mechanism (codegen.h). jit.cpp links the two with
// nvJitLink into one module per mechanism and launches the kernels from it.
// The step loops, stages, norm, controller and projection are the shared
// device functions of rosenbrock.cuh; the evaluations, the factorization and
// the solves are the mechanism's.
//
// One block per group: a team of 1 to 16 warps (blockDim = 32 x warps), every
// warp holding the group's cells in its 32 lanes (the generated code's operand
// stride). At most 128 registers per thread, so that sixteen warps are
// resident per SM whatever the team's size; jit.cpp chooses it by the number
// of blocks. Where the groups are too few even for one SM each, a cluster of
// sixteen-warp blocks on several SMs works on a group (the integrator kernel
// without the queue).
#define FO_LINK_GENERATED 1

#include <cuda_runtime.h>

#include "adjoint.cuh"
#include "rosenbrock.cuh"

extern "C" __global__ void __launch_bounds__(32 * 16, 1) fo_generated_solve_kernel(fo::SolveParams p) {
  extern __shared__ double smem[];
  double* red = smem;       // 32 doubles
  fo::RoundPace pace;
  double* w = smem + 32;    // a cluster's partial sums
  const int slot = blockIdx.x / cluster_blocks();
  double* scr = p.scratch + (int64_t)slot * p.slot_doubles;
  fo::rounds_join(p.rounds, pace);
  if (p.queue == nullptr) {
    fo::solve_group(p, slot, scr, w, red, pace);
  } else {
    __shared__ int next;
    for (;;) {
      __syncthreads();
      if (fo::team_leader()) next = atomicAdd(p.queue, 1);
      __syncthreads();
      const int g = next;
      if (g >= p.ngroups) break;
      fo::solve_group(p, g, scr, w, red, pace);
    }
  }
  fo::rounds_leave(pace);
}

// Several mechanisms in one persistent launch (the generated form of
// solve_multi_kernel): items [starts[b], starts[b+1]) of the queue are the
// groups of batch b, whose parameters carry the mechanism's index in this
// module; each block integrates whatever group it pulls next.
extern "C" __global__ void __launch_bounds__(32 * 16, 1)
    fo_generated_multi_kernel(const fo::SolveParams* __restrict__ batches, int nb, const int32_t* __restrict__ starts,
                              int32_t* queue, double* scratch, int64_t slot_doubles) {
  extern __shared__ double smem[];
  double* red = smem;
  fo::RoundPace pace;
  double* w = smem + 32;
  double* scr = scratch + (int64_t)blockIdx.x * slot_doubles;
  __shared__ int next;
  __shared__ fo::SolveParams params;
  int current = -1;
  fo::rounds_join(batches[0].rounds, pace);   // the same words in every batch
  const int total = starts[nb];
  for (;;) {
    __syncthreads();
    if (fo::team_leader()) next = atomicAdd(queue, 1);
    __syncthreads();
    const int item = next;
    if (item >= total) break;
    int b = 0;
    while (b + 1 < nb && item >= starts[b + 1]) ++b;
    fo::load_batch_params(batches, b, current, params);
    fo::solve_group(params, item - starts[b], scr, w, red, pace);
  }
  fo::rounds_leave(pace);
}

// The discrete adjoint of one interval (adjoint.cuh) on the mechanism's
// generated factorization, solves and transposed solves.
extern "C" __global__ void __launch_bounds__(32 * 16, 1) fo_generated_adjoint_kernel(fo::AdjParams a) {
  extern __shared__ double smem[];
  fo::adjoint_group(a, smem);
}
