// FP64 3x3 block helpers shared by the device translation units (internal linkage in each).
// Multiplies and adds are explicitly rounded (never fused) and follow the reference's loop order
// (engine/src/bsr.cpp:13-87), so results are bitwise those of the reference's serial code.
#pragma once
#include <cuda_runtime.h>

namespace rsg {
namespace {

// ------------------------------------------------------------------ FP64 block arithmetic, reference order, unfused
__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }

// one row of a 3x3 block times a 3-vector, accumulated from zero left to right
__device__ __forceinline__ double dot3(const double* a, const double* x) {
    return da(da(dm(a[0], x[0]), dm(a[1], x[1])), dm(a[2], x[2]));
}

// engine/src/bsr.cpp:67-87 for nb = 3: Gauss-Jordan on [A | I], partial pivoting, singular below 1e-14 max|a|
__device__ bool invert3(double* a) {
    double m[3][6];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) { m[i][j] = a[i * 3 + j]; m[i][3 + j] = (i == j) ? 1.0 : 0.0; }
    double scale = 0;
#pragma unroll
    for (int i = 0; i < 9; ++i) scale = fmax(scale, fabs(a[i]));
    if (!(scale > 0) || !isfinite(scale)) return false;
    for (int k = 0; k < 3; ++k) {
        int pr = k;
        for (int i = k + 1; i < 3; ++i)
            if (fabs(m[i][k]) > fabs(m[pr][k])) pr = i;
        if (fabs(m[pr][k]) <= dm(1e-14, scale)) return false;
        if (pr != k)
            for (int j = 0; j < 6; ++j) { const double t = m[k][j]; m[k][j] = m[pr][j]; m[pr][j] = t; }
        const double inv = __ddiv_rn(1.0, m[k][k]);
        for (int j = 0; j < 6; ++j) m[k][j] = dm(m[k][j], inv);
        for (int i = 0; i < 3; ++i) {
            if (i == k || m[i][k] == 0.0) continue;
            const double f = m[i][k];
            for (int j = 0; j < 6; ++j) m[i][j] = ds(m[i][j], dm(f, m[k][j]));
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) a[i * 3 + j] = m[i][3 + j];
    return true;
}
// pivot inversion with the reference's regularisation of singular blocks (engine/src/bsr.cpp:204-212);
// returns 1 when the block had to be regularised
__device__ int invert_pivot3(double* d) {
    double tmp[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) tmp[e] = d[e];
    if (invert3(d)) return 0;
    double sc = 0;
#pragma unroll
    for (int e = 0; e < 9; ++e) sc = fmax(sc, fabs(tmp[e]));
    if (!(sc > 0) || !isfinite(sc)) sc = 1.0;
#pragma unroll
    for (int e = 0; e < 9; ++e) d[e] = tmp[e];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const double de = d[e * 4];
        d[e * 4] = da(de, da(dm(de >= 0 ? 1e-8 : -1e-8, sc), de == 0 ? dm(sc, 1e-8) : 0.0));
    }
    if (!invert3(d)) {
#pragma unroll
        for (int e = 0; e < 9; ++e) d[e] = 0;
        const double inv = __ddiv_rn(1.0, sc);
        d[0] = inv; d[4] = inv; d[8] = inv;
    }
    return 1;
}

__device__ __forceinline__ void store9(double* p, const double* a) {
#pragma unroll
    for (int e = 0; e < 9; ++e) p[e] = a[e];
}
__device__ __forceinline__ void load9_ro(const double* p, double* a) {
#pragma unroll
    for (int e = 0; e < 9; ++e) a[e] = __ldg(p + e);
}

// one row of a 3x3 block (factor type TF) times a 3-vector of type TV, accumulated from zero left to right
__device__ __forceinline__ double rdot(const double* a, const double* x) { return da(da(dm(a[0], x[0]), dm(a[1], x[1])), dm(a[2], x[2])); }
__device__ __forceinline__ double rdot(const float* a, const double* x) {
    return da(da(dm(double(a[0]), x[0]), dm(double(a[1]), x[1])), dm(double(a[2]), x[2]));
}
__device__ __forceinline__ float rdot(const float* a, const float* x) {
    float s = 0.f;
    s += a[0] * x[0];
    s += a[1] * x[1];
    s += a[2] * x[2];
    return s;
}
__device__ __forceinline__ double vsub(double a, double b) { return ds(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }

}  // namespace
}  // namespace rsg
