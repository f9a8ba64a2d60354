// The Rosenbrock tableaus in the transformed form (fastode/tableaus.py:70-90),
// shared by the launch code and the generated integrator, whose stages are
// compiled for each.
#pragma once

#include "device.cuh"
#include "fastode_gb300.h"

namespace fo {

#ifdef __CUDACC__
__host__ __device__
#endif
constexpr DevTableau tableau_of(int id) {
  return id == FO_TABLEAU_ROS3
             ? DevTableau{0.43586652150845899941601945119356,
                          3,
                          {{0, 0, 0, 0}, {1.0, 0, 0, 0}, {1.0, 0.0, 0, 0}, {0, 0, 0, 0}},
                          {{0, 0, 0, 0},
                           {-0.10156171083877702091975600115545e01, 0, 0, 0},
                           {0.40759956452537699824805835358067e01, 0.92076794298330791242156818474003e01, 0, 0},
                           {0, 0, 0, 0}},
                          {1.0, 0.61697947043828245592553615689730e01, -0.42772256543218573326238373806514, 0},
                          {0.5, -0.29079558716805469821718236208017e01, 0.22354069897811569627360909276199, 0},
                          {1, 1, 0, 0}}
             : DevTableau{0.5,
                          4,
                          {{0, 0, 0, 0}, {0.0, 0, 0, 0}, {2.0, 0.0, 0, 0}, {2.0, 0.0, 1.0, 0}},
                          {{0, 0, 0, 0}, {4.0, 0, 0, 0}, {1.0, -1.0, 0, 0}, {1.0, -1.0, -8.0 / 3.0, 0}},
                          {2.0, 0.0, 1.0, 1.0},
                          {0.0, 0.0, 0.0, 1.0},
                          {1, 0, 1, 1}};
}

}  // namespace fo
