// The band of cells that boundary saving keeps, and its storage formats.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace pam {

// The saved band: the outer four rows and columns of the physical region
// (src/Migration.py:288-298), as a flat list - rows [N, N+4) and
// [N+nz-4, N+nz) over the nx physical columns, then columns [N, N+4) and
// [N+nx-4, N+nx) over the nz-8 rows in between.  Four cells is the stencil
// half-width, so the reverse steps of the cells inside the band read only the
// band and themselves.
__host__ __device__ inline long long band_cells(int nzi, int nxi) { return 8LL * nxi + 8LL * (nzi - 8); }

__device__ __forceinline__ void band_cell(long long i, int N, int nzi, int nxi, int& z, int& x) {
    const long long rows = 4LL * nxi;
    if (i < rows) { z = N + (int)(i / nxi); x = N + (int)(i % nxi); return; }
    i -= rows;
    if (i < rows) { z = N + nzi - 4 + (int)(i / nxi); x = N + (int)(i % nxi); return; }
    i -= rows;
    const long long side = 4LL * (nzi - 8);
    if (i < side) { z = N + 4 + (int)(i / 4); x = N + (int)(i % 4); return; }
    i -= side;
    z = N + 4 + (int)(i / 4);
    x = N + nxi - 4 + (int)(i % 4);
}

constexpr int kBandChunk = 256;   // cells per scale (one block)

template <typename T>
__device__ __forceinline__ T band_pack(float v);
template <>
__device__ __forceinline__ float band_pack<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 band_pack<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half band_pack<__half>(float v) { return __float2half_rn(v); }
__device__ __forceinline__ float band_unpack(float v) { return v; }
__device__ __forceinline__ float band_unpack(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float band_unpack(__half v) { return __half2float(v); }

}  // namespace pam
