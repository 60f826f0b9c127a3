// Whole FP64 Lanczos basis of one vector in one cooperative launch
// (plain_lanczos.cu); interface used by krylov.cu.
#pragma once

#include "common.cuh"

namespace rpm {

// Device scalars of a plain basis build (SLOT_SMALL).
struct LanczosScalars {
  unsigned counter[8];
  unsigned barrier, exits;  // grid barrier of the one-launch build (zero between launches)
  int stop;       // basis size after a breakdown (0 = running, -1 = zero vector)
  int timeout;    // nonzero: a grid barrier gave up
  double norm;    // ||state||
  double2 h1[RPM_MAX_KRYLOV];
  double2 h2[RPM_MAX_KRYLOV];
};

// Launches the build; false (nothing launched) when the system's layout or
// size is outside what the kernel covers.
bool launch_plain_basis(rpm_system* sys, const double2* state, int m, double tol, double2* basis, double* alpha,
                        double* beta, LanczosScalars* sc, cudaStream_t stream);

}  // namespace rpm
