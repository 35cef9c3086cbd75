// tri_index.cuh -- function qualifiers of the code that host and device share.
#pragma once

#ifdef __CUDACC__
#define EFMM_HD __host__ __device__ __forceinline__
#else
#define EFMM_HD inline
#endif
