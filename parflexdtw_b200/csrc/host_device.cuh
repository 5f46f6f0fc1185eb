// Qualifiers of functions that headers share with the host's own compiler.
#pragma once
#ifdef __CUDACC__
#define PFX_HD __host__ __device__ __forceinline__
#else
#define PFX_HD inline
#endif
