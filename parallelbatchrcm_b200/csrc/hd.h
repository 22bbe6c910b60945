// hd.h -- marks functions that device code and host code (or a host test)
// both compile: PBRCM_HD for either side, PBRCM_DEV for those that nvcc
// compiles for the device alone (they call device functions there).
#pragma once

#if defined(__CUDACC__)
#define PBRCM_HD __host__ __device__
#define PBRCM_DEV __device__ __forceinline__
#else
#define PBRCM_HD
#define PBRCM_DEV inline
#endif
