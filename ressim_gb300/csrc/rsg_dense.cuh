// Dense LU with partial pivoting of a small matrix by one thread block (AMG::factorCoarsest, engine/src/amg.cpp:273-295),
// shared by the device translation units (internal linkage in each).
//
// The elimination is a chain of m steps (pivot, interchange, scaled column, rank-1 update), each with its synchronisations, so
// a step keeps to three barriers: the pivot's winner is reduced by every warp on its own, the interchange and the scaled
// column go with the copies of row k and column k that the update reads, and the update is a warp per row. The matrix stays in
// shared memory when it fits (m <= 160 in FP64, 226 in FP32). Beyond about 150 rows the FP64 form is bound by the FP64 pipe
// of its SM (2/3 m^3 operations at two a clock).
// Every element takes the reference's operations in its order.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "rsg_impl.h"

namespace rsg {
namespace {

constexpr int kDenseThreads = 1024;
constexpr int kDenseMax = 1024;              // rows at most (the hierarchy keeps a coarsest level dense up to 800)

__device__ __forceinline__ double lmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double lsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ldiv_(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float lmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float lsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float ldiv_(float a, float b) { return __fdiv_rn(a, b); }
template <class T> __device__ __forceinline__ T lu_tiny();
template <> __device__ __forceinline__ double lu_tiny<double>() { return 1e-300; }
template <> __device__ __forceinline__ float lu_tiny<float>() { return 1.17549435e-38f; }   // smallest normal float

// dynamic shared memory of a launch whose largest matrix has m rows (0: it stays in global memory)
template <class T>
unsigned dense_lu_smem(int m) {
    const size_t need = size_t(m) * size_t(m) * sizeof(T);
    return need <= 200 * 1024 ? unsigned(need) : 0u;
}
template <class T>
__device__ __forceinline__ T* dense_lu_place(int m, unsigned smemBytes, unsigned char* sm, T* global) {
    return size_t(m) * size_t(m) * sizeof(T) <= smemBytes ? reinterpret_cast<T*>(sm) : global;
}

// a (m x m, row-major, shared or global) factored in place, piv[k] = the row interchanged with row k. kDenseThreads threads.
template <class T>
__device__ __noinline__ void dense_lu(int m, T* a, int* piv) {
    __shared__ T bestV[32];
    __shared__ int bestI[32];
    __shared__ T urow[kDenseMax], lcol[kDenseMax];
    const int tid = int(threadIdx.x), lane = tid & 31, wid = tid >> 5, nw = int(blockDim.x) >> 5;
    for (int k = 0; k < m; ++k) {
        // the first row i >= k of the largest |a_ik| (the reference moves only on a strictly larger value)
        T best = T(-1);
        int bi = m;
        for (int i = k + tid; i < m; i += int(blockDim.x)) {
            const T v = fabs(a[size_t(i) * m + k]);
            if (v > best) { best = v; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { bestV[wid] = best; bestI[wid] = bi; }
        __syncthreads();
        best = lane < nw ? bestV[lane] : T(-1);
        bi = lane < nw ? bestI[lane] : m;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        const T akk = a[size_t(k) * m + k];
        const int pr = best > fabs(akk) ? bi : k;
        T dk = a[size_t(pr) * m + k];
        if (fabs(dk) < lu_tiny<T>()) dk = lu_tiny<T>();
        // column k below the pivot, scaled (row pr holds row k's entry after the interchange), and row k
        for (int t = tid; t < m; t += int(blockDim.x)) {
            if (t > k) lcol[t] = ldiv_(t == pr ? akk : a[size_t(t) * m + k], dk);
            urow[t] = t == k ? dk : a[size_t(pr) * m + t];
        }
        if (tid == 0) piv[k] = pr;
        __syncthreads();
        for (int t = tid; t < m; t += int(blockDim.x)) {
            if (pr != k && t != k) a[size_t(pr) * m + t] = a[size_t(k) * m + t];
            a[size_t(k) * m + t] = urow[t];
            if (t > k) a[size_t(t) * m + k] = lcol[t];
        }
        __syncthreads();
        for (int i = k + 1 + wid; i < m; i += nw) {
            const T f = lcol[i];
            if (f != T(0))
                for (int j = k + 1 + lane; j < m; j += 32) a[size_t(i) * m + j] = lsub(a[size_t(i) * m + j], lmul(f, urow[j]));
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace rsg
