// hd.h -- functions of kernels that also compile for the CPU (their tests).
#pragma once

#ifdef __CUDACC__
#define GS_HD __host__ __device__ __forceinline__
#else
#define GS_HD inline
#endif
