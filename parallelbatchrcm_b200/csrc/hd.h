// hd.h -- marks functions that device code and host code (or a host test)
// both compile.
#pragma once

#if defined(__CUDACC__)
#define PBRCM_HD __host__ __device__
#else
#define PBRCM_HD
#endif
