// Dense LU with partial pivoting of a small matrix by a cluster of thread blocks or by one block (AMG::factorCoarsest,
// engine/src/amg.cpp:273-295), shared by the device translation units (internal linkage in each).
//
// One block is bound by the FP64 pipe of its SM (2/3 m^3 operations at two a clock: 2.7 ms at 256 rows). So the columns are
// dealt out over a cluster of eight blocks, each holding its columns in shared memory (in global memory beyond 424 rows
// in FP64, 600 in FP32). Step k: the interchange and the rank-1 update of a block's own columns; the owner of column k + 1 updates
// that one first, finds its pivot and sends the scaled column to every block's shared memory, so that a step has one
// cluster barrier. 256 rows, FP64: 2.7 -> 1.45 ms. Where many matrices fill the GPU by themselves a block takes one alone
// (rsg_cpr.cu has the rule). Every element takes the reference's operations in its order.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "rsg_impl.h"

namespace rsg {
namespace {

// CL blocks of NT threads take a matrix: the cluster, or (rsg_cpr.cu: small matrices, and batches of many) one block
constexpr int kDenseCluster = 8, kDenseThreads = 512;
// shared memory for a block's columns; a single block leaves room for others on its SM (1,000 matrices of 100 rows in FP64, a set-up:
// 4.28 ms with them on chip, 3.54 ms not)
template <int CL> constexpr size_t kDenseSmem = CL > 1 ? 176 * 1024 : 40 * 1024;
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
template <int CL> __host__ __device__ constexpr int dense_cols(int m) { return (m + CL - 1) / CL; }
template <class T, int CL>
unsigned dense_lu_smem(int m) {
    const size_t need = size_t(m) * size_t(dense_cols<CL>(m)) * sizeof(T);
    return need <= kDenseSmem<CL> ? unsigned(need) : 0u;
}

// the columns j = c * CL + rank of a matrix, as this block holds them
template <class T, int CL>
struct DenseCols {
    T* a;
    int m, rank, nc, rs, cs;                 // columns held, strides of a row and of a column
    bool onchip;
    __device__ T& at(int i, int c) const { return a[size_t(i) * rs + size_t(c) * cs]; }
};
template <class T, int CL>
__device__ __forceinline__ DenseCols<T, CL> dense_place(int m, int rank, unsigned smemBytes, unsigned char* sm, T* lu) {
    const int ld = dense_cols<CL>(m), nc = m > rank ? (m - rank + CL - 1) / CL : 0;
    if (size_t(m) * size_t(ld) * sizeof(T) <= smemBytes) return {reinterpret_cast<T*>(sm), m, rank, nc, ld, 1, true};
    return {lu + rank, m, rank, nc, m, CL, false};
}
template <int CL>
__device__ __forceinline__ int cluster_rank() {
    if constexpr (CL == 1) return 0;
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return int(r);
}
template <int CL>
__device__ __forceinline__ void cluster_sync() {
    if constexpr (CL == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same variable in the shared memory of another block of the cluster
template <class T>
__device__ __forceinline__ T* cluster_peer(T* p, int rank) {
    unsigned long long out;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<unsigned long long>(p)), "r"(rank));
    return reinterpret_cast<T*>(out);
}

// this block's columns of the sparse matrix (rp, ci, v; rows and columns through perm), zero elsewhere
template <class T, int CL>
__device__ __forceinline__ void dense_fill(const DenseCols<T, CL>& D, const int* __restrict__ rp, const int* __restrict__ ci,
                                           const double* __restrict__ v, const int* __restrict__ perm) {
    const int tid = int(threadIdx.x), nt = int(blockDim.x);
    for (int q = tid; q < D.m * D.nc; q += nt) D.at(q / D.nc, q % D.nc) = T(0);
    __syncthreads();
    for (int k = tid; k < D.m; k += nt) {
        const int I = __ldg(perm + k);
        for (int p = __ldg(rp + k); p < __ldg(rp + k + 1); ++p) {
            const int J = __ldg(perm + __ldg(ci + p));
            if (J % CL == D.rank) D.at(I, J / CL) = T(v[p]);
        }
    }
    __syncthreads();
}
// and the factored columns to the m x m matrix in global memory
template <class T, int CL>
__device__ __forceinline__ void dense_out(const DenseCols<T, CL>& D, T* lu) {
    if (!D.onchip) return;
    for (int q = int(threadIdx.x); q < D.m * D.nc; q += int(blockDim.x))
        lu[size_t(q / D.nc) * D.m + size_t(q % D.nc) * CL + D.rank] = D.at(q / D.nc, q % D.nc);
}

// D factored in place over the CL blocks, piv[k] = the row interchanged with row k. NT threads; the columns are in
// place and visible to their own block.
template <int NT, class T, int CL>
__device__ __noinline__ void dense_lu(const DenseCols<T, CL>& D, int* piv) {
    __shared__ T bestV[NT / 32];
    __shared__ int bestI[NT / 32];
    __shared__ T lcol[2][kDenseMax];         // the scaled column of step k (in [k & 1]), sent by its owner
    __shared__ int prow[2];
    const int tid = int(threadIdx.x), lane = tid & 31, wid = tid >> 5, m = D.m;
    constexpr int NW = NT / 32;
    // pivot of column k (this block's), its scaled column into lcol[k & 1] of every block
    auto panel = [&](int k) {
        const int c = k / CL;
        // the first row i >= k of the largest |a_ik| (the reference moves only on a strictly larger value)
        T best = T(-1);
        int bi = m;
        for (int i = k + tid; i < m; i += NT) {
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
        T l[kDenseMax / NT];
#pragma unroll
        for (int u = 0; u < kDenseMax / NT; ++u) {   // (row pr holds row k's entry after the interchange)
            const int i = k + 1 + tid + u * NT;
            l[u] = i < m ? ldiv_(i == pr ? akk : D.at(i, c), dk) : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kDenseMax / NT; ++u) {
            const int i = k + 1 + tid + u * NT;
            if (i >= m) break;
            D.at(i, c) = l[u];
            if constexpr (CL == 1) lcol[k & 1][i] = l[u];
            else
                for (int r = 0; r < CL; ++r) *cluster_peer(&lcol[k & 1][i], r) = l[u];
        }
        if (tid == 0) {
            D.at(k, c) = dk;
            if constexpr (CL == 1) prow[k & 1] = pr;
            else
                for (int r = 0; r < CL; ++r) *cluster_peer(&prow[k & 1], r) = pr;
        }
    };
    cluster_sync<CL>();                      // every block has started
    if (D.rank == 0) panel(0);
    cluster_sync<CL>();
    for (int k = 0; k < m; ++k) {
        const T* lc = lcol[k & 1];
        const int pr = prow[k & 1], own = k % CL == D.rank ? k / CL : -1;
        if (pr != k)
            for (int c = tid; c < D.nc; c += NT)
                if (c != own) {                              // (column k is already in its final order)
                    const T t = D.at(k, c);
                    D.at(k, c) = D.at(pr, c);
                    D.at(pr, c) = t;
                }
        if (tid == 0 && D.rank == 0) piv[k] = pr;
        __syncthreads();
        int done = -1;                                       // the column of step k + 1, when it is this block's
        if (k + 1 < m && (k + 1) % CL == D.rank) {
            done = (k + 1) / CL;
            const T u = D.at(k, done);
            for (int i = k + 1 + tid; i < m; i += NT)
                if (lc[i] != T(0)) D.at(i, done) = lsub(D.at(i, done), lmul(lc[i], u));
            __syncthreads();
            panel(k + 1);
        }
        // the other columns beyond k: a lane per column, the warps over the rows
        const int c0 = k + 1 > D.rank ? (k + 1 - D.rank + CL - 1) / CL : 0;
        for (int cb = c0; cb < D.nc; cb += 32) {
            const int c = cb + lane;
            const bool act = c < D.nc && c != done;
            const T u = act ? D.at(k, c) : T(0);
            for (int i = k + 1 + wid; i < m; i += NW) {
                const T f = lc[i];
                if (f != T(0) && act) D.at(i, c) = lsub(D.at(i, c), lmul(f, u));
            }
        }
        cluster_sync<CL>();
    }
}

// launch of a dense factorisation: CL blocks per system
template <int CL, int NT, class K, class... A>
void launch_dense(K kernel, int nsys, unsigned smem, cudaStream_t st, A... args) {
    raise_smem_limit(reinterpret_cast<const void*>(kernel), int(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(nsys * CL));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace rsg
