// Dense LU with partial pivoting of a small matrix by a cluster of thread blocks (AMG::factorCoarsest,
// engine/src/amg.cpp:273-295), shared by the device translation units (internal linkage in each).
//
// One block is bound by the FP64 pipe of its SM (2/3 m^3 operations at two a clock: 2.7 ms at 256 rows). So the columns are
// dealt out over a cluster of eight blocks, each holding its columns in shared memory (in global memory beyond about 440
// rows in FP64). Step k: the interchange and the rank-1 update of a block's own columns; the owner of column k + 1 updates
// that one first, finds its pivot and sends the scaled column to every block's shared memory, so that a step has one
// cluster barrier. 256 rows, FP64: 2.7 -> 1.45 ms. Every element takes the reference's operations in its order.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "rsg_impl.h"

namespace rsg {
namespace {

constexpr int kDenseThreads = 512;
constexpr int kDenseCluster = 8;
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

// columns of a block, and the dynamic shared memory of a launch whose largest matrix has m rows (0: in global memory)
__host__ __device__ constexpr int dense_cols(int m) { return (m + kDenseCluster - 1) / kDenseCluster; }
template <class T>
unsigned dense_lu_smem(int m) {
    const size_t need = size_t(m) * size_t(dense_cols(m)) * sizeof(T);
    return need <= 176 * 1024 ? unsigned(need) : 0u;
}

// the columns j = c * kDenseCluster + rank of a matrix, as this block holds them
template <class T>
struct DenseCols {
    T* a;
    int m, rank, nc, rs, cs;                 // columns held, strides of a row and of a column
    __device__ T& at(int i, int c) const { return a[size_t(i) * rs + size_t(c) * cs]; }
};
template <class T>
__device__ __forceinline__ DenseCols<T> dense_place(int m, int rank, unsigned smemBytes, unsigned char* sm, T* lu) {
    const int ld = dense_cols(m), nc = m > rank ? (m - rank + kDenseCluster - 1) / kDenseCluster : 0;
    if (size_t(m) * size_t(ld) * sizeof(T) <= smemBytes) return {reinterpret_cast<T*>(sm), m, rank, nc, ld, 1};
    return {lu + rank, m, rank, nc, m, kDenseCluster};
}
__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return int(r);
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same variable in the shared memory of another block of the cluster
template <class T>
__device__ __forceinline__ T* cluster_peer(T* p, int rank) {
    unsigned long long out;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<unsigned long long>(p)), "r"(rank));
    return reinterpret_cast<T*>(out);
}

// this block's columns of the sparse matrix (rp, ci, v; rows and columns through perm), zero elsewhere
template <class T>
__device__ __forceinline__ void dense_fill(const DenseCols<T>& D, const int* __restrict__ rp, const int* __restrict__ ci,
                                           const double* __restrict__ v, const int* __restrict__ perm) {
    const int tid = int(threadIdx.x), nt = int(blockDim.x);
    for (int q = tid; q < D.m * D.nc; q += nt) D.at(q / D.nc, q % D.nc) = T(0);
    __syncthreads();
    for (int k = tid; k < D.m; k += nt) {
        const int I = __ldg(perm + k);
        for (int p = __ldg(rp + k); p < __ldg(rp + k + 1); ++p) {
            const int J = __ldg(perm + __ldg(ci + p));
            if (J % kDenseCluster == D.rank) D.at(I, J / kDenseCluster) = T(v[p]);
        }
    }
    __syncthreads();
}
// and the factored columns to the m x m matrix in global memory
template <class T>
__device__ __forceinline__ void dense_out(const DenseCols<T>& D, T* lu) {
    if (D.cs == kDenseCluster) return;
    for (int q = int(threadIdx.x); q < D.m * D.nc; q += int(blockDim.x))
        lu[size_t(q / D.nc) * D.m + size_t(q % D.nc) * kDenseCluster + D.rank] = D.at(q / D.nc, q % D.nc);
}

// D factored in place over the cluster, piv[k] = the row interchanged with row k. kDenseThreads threads; the columns are in
// place and visible to their own block.
template <class T>
__device__ __noinline__ void dense_lu(const DenseCols<T>& D, int* piv) {
    __shared__ T bestV[kDenseThreads / 32];
    __shared__ int bestI[kDenseThreads / 32];
    __shared__ T lcol[2][kDenseMax];         // the scaled column of step k (in [k & 1]), sent by its owner
    __shared__ int prow[2];
    const int tid = int(threadIdx.x), lane = tid & 31, wid = tid >> 5, m = D.m;
    constexpr int NW = kDenseThreads / 32;
    // pivot of column k (this block's), its scaled column into lcol[k & 1] of every block
    auto panel = [&](int k) {
        const int c = k / kDenseCluster;
        // the first row i >= k of the largest |a_ik| (the reference moves only on a strictly larger value)
        T best = T(-1);
        int bi = m;
        for (int i = k + tid; i < m; i += kDenseThreads) {
            const T v = fabs(D.at(i, c));
            if (v > best) { best = v; bi = i; }
        }
        auto reduce = [&]() {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const T ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
        };
        reduce();
        if (lane == 0) { bestV[wid] = best; bestI[wid] = bi; }
        __syncthreads();
        best = lane < NW ? bestV[lane] : T(-1);
        bi = lane < NW ? bestI[lane] : m;
        reduce();
        const T akk = D.at(k, c);
        const int pr = best > fabs(akk) ? bi : k;
        T dk = D.at(pr, c);
        if (fabs(dk) < lu_tiny<T>()) dk = lu_tiny<T>();
        T l[kDenseMax / kDenseThreads];
#pragma unroll
        for (int u = 0; u < kDenseMax / kDenseThreads; ++u) {   // (row pr holds row k's entry after the interchange)
            const int i = k + 1 + tid + u * kDenseThreads;
            l[u] = i < m ? ldiv_(i == pr ? akk : D.at(i, c), dk) : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kDenseMax / kDenseThreads; ++u) {
            const int i = k + 1 + tid + u * kDenseThreads;
            if (i >= m) break;
            D.at(i, c) = l[u];
            for (int r = 0; r < kDenseCluster; ++r) *cluster_peer(&lcol[k & 1][i], r) = l[u];
        }
        if (tid == 0) {
            D.at(k, c) = dk;
            for (int r = 0; r < kDenseCluster; ++r) *cluster_peer(&prow[k & 1], r) = pr;
        }
    };
    cluster_sync();                          // every block has started
    if (D.rank == 0) panel(0);
    cluster_sync();
    for (int k = 0; k < m; ++k) {
        const T* lc = lcol[k & 1];
        const int pr = prow[k & 1], own = k % kDenseCluster == D.rank ? k / kDenseCluster : -1;
        if (pr != k)
            for (int c = tid; c < D.nc; c += kDenseThreads)
                if (c != own) {                              // (column k is already in its final order)
                    const T t = D.at(k, c);
                    D.at(k, c) = D.at(pr, c);
                    D.at(pr, c) = t;
                }
        if (tid == 0 && D.rank == 0) piv[k] = pr;
        __syncthreads();
        int done = -1;                                       // the column of step k + 1, when it is this block's
        if (k + 1 < m && (k + 1) % kDenseCluster == D.rank) {
            done = (k + 1) / kDenseCluster;
            const T u = D.at(k, done);
            for (int i = k + 1 + tid; i < m; i += kDenseThreads)
                if (lc[i] != T(0)) D.at(i, done) = lsub(D.at(i, done), lmul(lc[i], u));
            __syncthreads();
            panel(k + 1);
        }
        // the other columns beyond k: a lane per column, the warps over the rows
        const int c0 = k + 1 > D.rank ? (k + 1 - D.rank + kDenseCluster - 1) / kDenseCluster : 0;
        for (int cb = c0; cb < D.nc; cb += 32) {
            const int c = cb + lane;
            const bool act = c < D.nc && c != done;
            const T u = act ? D.at(k, c) : T(0);
            for (int i = k + 1 + wid; i < m; i += NW) {
                const T f = lc[i];
                if (f != T(0) && act) D.at(i, c) = lsub(D.at(i, c), lmul(f, u));
            }
        }
        cluster_sync();
    }
}

// cluster launch of a dense factorisation: kDenseCluster blocks per system
template <class K, class... A>
void launch_dense(K kernel, int nsys, unsigned smem, cudaStream_t st, A... args) {
    raise_smem_limit(reinterpret_cast<const void*>(kernel), int(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(nsys * kDenseCluster));
    cfg.blockDim = dim3(kDenseThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kDenseCluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace rsg
