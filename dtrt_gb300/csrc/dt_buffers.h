// dtrt_gb300 — device buffers that grow on demand, and what gives way when the device is full.
#pragma once
#include <algorithm>

#include <cuda_runtime_api.h>

namespace dt {

// A buffer of at least `need` bytes at *ptr (its contents are not kept). Where the device has no
// room, the spare buffer, which a render can do without, is freed and the allocation tried again.
inline cudaError_t grow_buffer(void **ptr, size_t *have, size_t need, void **spare, size_t *spare_have) {
    if (*have >= need && *ptr) return cudaSuccess;
    if (*ptr) cudaFree(*ptr);
    *ptr = nullptr;
    *have = 0;
    need = std::max<size_t>(need, 256);
    cudaError_t e = cudaMalloc(ptr, need);
    if (e != cudaSuccess && spare != ptr && *spare) {
        cudaGetLastError();
        cudaFree(*spare);
        *spare = nullptr;
        *spare_have = 0;
        e = cudaMalloc(ptr, need);
    }
    if (e != cudaSuccess) *ptr = nullptr;
    else *have = need;
    return e;
}

// reserve(k) makes the workspaces of k lanes, drop() frees what a failed attempt has made: the
// lanes that could be had, `lanes` or else 1, and 0 (the error cleared) when the device has no
// room for one.
template <class F, class D>
int fit_lanes(int lanes, F reserve, D drop) {
    for (int k = lanes; k >= 1; k = k > 1 ? 1 : 0) {
        if (reserve(k)) return k;
        cudaGetLastError();
        drop();
    }
    return 0;
}

}  // namespace dt
