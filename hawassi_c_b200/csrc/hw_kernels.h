// hw_kernels.h -- host-callable launchers of the per-slice-size kernels.
#pragma once

#include <cuda_runtime.h>

#include "hw_device.cuh"

#define HW_DECLARE(MM)                                                                             \
  cudaError_t hw_attr_##MM();                                                                      \
  /* mode 0 run, 1 one step, of the nmem listed members; with a queue, ngrid clusters pull them */ \
  cudaError_t hw_evolve_##MM(int mode, hwdev::DevMember* mems, const int* list, int nmem, int C, \
                             cudaStream_t s, int* queue, int ngrid);                              \
  cudaError_t hw_rhs_##MM(hwdev::DevMember* mems, int mi, int C, double t, const double* y,       \
                          double* dy, double2* scratch, cudaStream_t s);                          \
  int hw_max_clusters_##MM(int C);
HW_DECLARE(256)
HW_DECLARE(512)
HW_DECLARE(1024)
HW_DECLARE(2048)
#undef HW_DECLARE
