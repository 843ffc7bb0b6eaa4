// Device kernels of the rsg solver (sm_103a).
//
// * BILU0 factorisation and the forward / backward sweeps are exact natural-order ILU(0): rows are processed in
//   a level order (a topological order of the L, resp. U, dependencies) by a persistent grid whose warps claim
//   rows from an atomic counter; a row waits for the rows it depends on, in the sweeps on their values themselves, in
//   the factorisation through per-row flags (rsg_sync.cuh). Claiming in order
//   guarantees that every awaited row belongs to a warp that is already running, so the waits always end; each
//   wait is additionally bounded and reports RSG_ETIMEOUT.
// * FP64 block arithmetic uses explicitly rounded multiplies and adds in the reference's loop order
//   (engine/src/bsr.cpp:13-64), so factors, sweeps and SpMV are bitwise those of the reference's serial code.
// * Tile kernels (SpMV, vector updates) cover TILE_ROWS block rows of one system with 3 threads per block row;
//   inner products are reduced per tile and then, in the last tile to finish, per system in a fixed order
//   (deterministic), and the BiCGSTAB scalar recurrences are evaluated on the device.
#include "rsg_impl.h"
#include "rsg_block3.cuh"
#include "rsg_reduce.cuh"
#include "rsg_sync.cuh"

#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <type_traits>

namespace rsg {

namespace {

constexpr int kSweepThreads = 128;

// ------------------------------------------------------------------ BILU0 factorisation (sync-free, level order)
// engine/src/bsr.cpp:183-215 row by row; rows of a system claimed in forward level order. W: arithmetic of the
// elimination, F: storage of the factors. (double, double) is the reference's FP64 factorisation; (double, float) the
// lean one (engine/src/bsr.cpp:219-263: the row, rounded to float, eliminated in double against the float factors of
// earlier rows, then rounded); (float, float) the precision form's FP32 elimination. The pivot block is inverted in FP64.
//
// A warp takes one row. What bounds the factorisation is its chain of dependent rows -- a level of the stencil, or a well
// clique of 30-40 rows that each eliminate against all the earlier ones -- so the work of one row is spread over the
// lanes: the row lives in shared memory, nine lanes form the block L_ik, 27 lanes update three target blocks at a time
// (one element each, the reference's operations in its order), six lanes hold the columns of [D | I] in the inversion, and
// the blocks of the next entry are on their way while one is eliminated. A thread per row paid every block's loads and
// arithmetic one after another: 180,000 rows with four 30-layer wells 28 -> 3.4 ms, 277,000 rows with five 42-layer wells
// (lean) 115 -> 11.9 ms, 11,200 rows 2.82 -> 0.57 ms; FP32, a block per system before, 11,200 rows 2.4 -> 0.47 ms, 64 systems
// 3.29 -> 2.95 ms.
__device__ __forceinline__ double fmul(double a, double b) { return dm(a, b); }
__device__ __forceinline__ double fadd(double a, double b) { return da(a, b); }
__device__ __forceinline__ double fsub(double a, double b) { return ds(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }

// Inversion of a pivot block by a warp: lane j < 6 holds column j of [D | I]; invert3's operations in its order
// (rsg_block3.cuh), so the same bits. The result of D^-1 element (i, j) is in out[i] of lane 3 + j. False (every lane): a
// singular or non-finite block.
template <class W>
__device__ __forceinline__ bool warp_invert3(const W* D, int lane, double (&out)[3]) {
    double m[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) m[i] = lane < 3 ? double(D[3 * i + lane]) : (lane == 3 + i ? 1.0 : 0.0);
    double sc = lane < 3 ? fmax(fmax(fmax(0.0, fabs(m[0])), fabs(m[1])), fabs(m[2])) : 0.0;
    sc = fmax(fmax(__shfl_sync(0xffffffffu, sc, 0), __shfl_sync(0xffffffffu, sc, 1)), __shfl_sync(0xffffffffu, sc, 2));
    if (!(sc > 0) || !isfinite(sc)) return false;
    const double thr = dm(1e-14, sc);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double c[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) c[i] = __shfl_sync(0xffffffffu, m[i], k);
        int pr = k;
        double big = fabs(c[k]), cp = c[k];
#pragma unroll
        for (int i = k + 1; i < 3; ++i)
            if (fabs(c[i]) > big) { pr = i; big = fabs(c[i]); cp = c[i]; }
        if (big <= thr) return false;
#pragma unroll
        for (int i = k + 1; i < 3; ++i)
            if (pr == i) {
                const double t = m[k], u = c[k];
                m[k] = m[i]; m[i] = t;
                c[k] = c[i]; c[i] = u;
            }
        m[k] = dm(m[k], __ddiv_rn(1.0, cp));
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i != k && c[i] != 0.0) m[i] = ds(m[i], dm(c[i], m[k]));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = m[i];
    return true;
}

template <class W, class F>
__global__ void __launch_bounds__(kSweepThreads) k_factor(int n, int chunk, const int* __restrict__ rowPtr, const int* __restrict__ col,
                                                          const int* __restrict__ diag, const int* __restrict__ ford,
                                                          const int* __restrict__ elimPtr, const int* __restrict__ elimT,
                                                          const int* __restrict__ elimQ, const double* __restrict__ val, F* lu, W* work,
                                                          int* flagL, int epoch, unsigned* ctr, int* nreg, int* err) {
    __shared__ W rows[kSweepThreads / 32][kFacRow * 9];
    const int lane = threadIdx.x & 31;
    const unsigned all = 0xffffffffu;
    const int g = lane / 9, el = lane % 9, er = el / 3, ec = el % 3;   // this lane's target of three, and element
    int at = 0, end = 0;
    for (;;) {
        if (at >= end) {                                      // the next `chunk` rows of the claim order
            unsigned got = 0;
            if (lane == 0) got = atomicAdd(ctr, unsigned(chunk));
            at = int(__shfl_sync(all, got, 0));
            end = min(n, at + chunk);
            if (at >= n) break;
        }
        const int i = __ldg(ford + at++);
        const int r0 = __ldg(rowPtr + i), r1 = __ldg(rowPtr + i + 1), d = __ldg(diag + i);
        W* row = (r1 - r0) <= kFacRow ? rows[threadIdx.x >> 5] : work + size_t(r0) * 9;
        for (int e = lane; e < 9 * (r1 - r0); e += 32) row[e] = W(F(__ldg(val + size_t(r0) * 9 + e)));
        for (int c0 = r0; c0 < d; c0 += 32) {                 // the entries before the diagonal, 32 at a time
            const int cn = min(32, d - c0);
            int k = 0, dk = 0, q0 = 0, q1 = 0;                // this lane's entry: column, its pivot block, its eliminations
            if (lane < cn) {
                k = __ldg(col + c0 + lane);
                dk = __ldg(diag + k);
                q0 = __ldg(elimPtr + c0 + lane);
                q1 = __ldg(elimPtr + c0 + lane + 1);
            }
            {                                                 // wait for the rows of the chunk (bounded)
                bool pending = lane < cn;
                unsigned ns = 0;
                for (unsigned it = 0;; ++it) {
                    if (pending && ld_relaxed(flagL + k) == epoch) pending = false;
                    if (!__any_sync(all, pending)) break;
                    if (it >= 64) {
                        __nanosleep(ns);
                        ns = ns < 32 ? 32 : (ns < 256 ? 2 * ns : 256);
                        bool stop = (it & 255u) == 255u && *(volatile int*)err != 0;
                        if (it >= 64 + kSpinLimit) { if (pending) atomicOr(err, ERR_TIMEOUT); stop = true; }
                        if (__any_sync(all, stop)) break;     // (the lanes leave together: they may read *err differently)
                    }
                }
            }
            fence_acquire();
            __syncwarp();
            // blocks of an entry: column ec of U_kk (lanes 0-8) and of the first three targets' U_kq (27 lanes)
            W u[3], U[3];
            int t = -1;
            auto fetch = [&](int p, W (&pu)[3], W (&pU)[3], int& pt) {
                const int pd = __shfl_sync(all, dk, p), a0 = __shfl_sync(all, q0, p), a1 = __shfl_sync(all, q1, p);
                pt = -1;
                if (lane < 27 && a0 + g < a1) {
                    pt = __ldg(elimT + a0 + g) - r0;
                    const F* f = lu + size_t(__ldg(elimQ + a0 + g)) * 9 + ec;
#pragma unroll
                    for (int m = 0; m < 3; ++m) pU[m] = W(f[3 * m]);
                }
                if (lane < 9) {
                    const F* f = lu + size_t(pd) * 9 + ec;
#pragma unroll
                    for (int m = 0; m < 3; ++m) pu[m] = W(f[3 * m]);
                }
            };
            fetch(0, u, U, t);
            for (int p = 0; p < cn; ++p) {
                W un[3], Un[3];
                int tn = -1;
                if (p + 1 < cn) fetch(p + 1, un, Un, tn);     // the next entry's blocks (final rows: nothing here changes them)
                const int a0 = __shfl_sync(all, q0, p), a1 = __shfl_sync(all, q1, p);
                W* L = row + size_t(c0 - r0 + p) * 9;
                W l = W(0);                                   // L_ik = A_ik U_kk^-1
                if (lane < 9) {
#pragma unroll
                    for (int m = 0; m < 3; ++m) l = fadd(l, fmul(L[3 * er + m], u[m]));
                }
                __syncwarp();
                if (lane < 9) L[el] = l;
                __syncwarp();
                W Lr[3];
#pragma unroll
                for (int m = 0; m < 3; ++m) Lr[m] = L[3 * er + m];
                auto elim = [&](int tt, const W (&uu)[3]) {    // A_it -= L_ik U_kq, one element
                    W s = W(0);
#pragma unroll
                    for (int m = 0; m < 3; ++m) s = fadd(s, fmul(Lr[m], uu[m]));
                    row[size_t(tt) * 9 + el] = fsub(row[size_t(tt) * 9 + el], s);
                };
                if (t >= 0) elim(t, U);
                for (int q = a0 + 3 + g; q - g < a1; q += 12) {   // further targets: the loads of twelve at once
                    W V[4][3];
                    int tt[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        tt[v] = -1;
                        if (lane < 27 && q + 3 * v < a1) {
                            tt[v] = __ldg(elimT + q + 3 * v) - r0;
                            const F* f = lu + size_t(__ldg(elimQ + q + 3 * v)) * 9 + ec;
#pragma unroll
                            for (int m = 0; m < 3; ++m) V[v][m] = W(f[3 * m]);
                        }
                    }
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        if (tt[v] >= 0) elim(tt[v], V[v]);
                }
                __syncwarp();
#pragma unroll
                for (int m = 0; m < 3; ++m) { u[m] = un[m]; U[m] = Un[m]; }
                t = tn;
            }
        }
        __syncwarp();
        W* D = row + size_t(d - r0) * 9;
        double inv[3];
        if (warp_invert3(D, lane, inv)) {
            __syncwarp();
            if (lane >= 3 && lane < 6)
#pragma unroll
                for (int m = 0; m < 3; ++m) D[3 * m + lane - 3] = W(inv[m]);
        } else {                                              // the reference's regularised inverse
            __syncwarp();
            if (lane == 0) {
                double B[9];
#pragma unroll
                for (int e = 0; e < 9; ++e) B[e] = double(D[e]);
                if (invert_pivot3(B)) atomicAdd(nreg, 1);
#pragma unroll
                for (int e = 0; e < 9; ++e) D[e] = W(B[e]);
            }
        }
        __syncwarp();
        for (int e = lane; e < 9 * (r1 - r0); e += 32) lu[size_t(r0) * 9 + e] = F(row[e]);
        __syncwarp();                                         // (orders the lanes' stores before the release)
        if (lane == 0) st_release(flagL + i, epoch);
    }
}

// The same elimination by a thread per row, for levels so wide that a warp per row is bound by its FP64 instructions (the
// inversion of a row's pivot block costs a warp what it costs 32 rows here): rows of at most kLaneRow blocks, held in local
// memory. The line is at 70 rows of a level per SM, 30 where the elimination is FP32 and the inversion most of the FP64 work; a warp
// per row / a thread per row (/ the former kernels), FP64: 152 systems of 2,500 rows (7,900 rows a level) 2.28 / 2.69 (2.60) ms,
// 300 of 1,000 (10,700) 1.79 / 1.57 (1.61), 300 of 3,300 (22,000) 5.90 / 4.25 (4.22); FP32 factors of FP64 rows: 7.26 / 5.31 (5.52);
// FP32: 64 of 2,500 (3,300) 0.73 / 0.90 (0.87), 300 of 400 (5,500) 0.53 / 0.46 (0.54), 300 of 3,300 4.17 / 1.51 (2.22).
constexpr int kLaneRow = 8;
template <class W, class F>
__global__ void __launch_bounds__(kSweepThreads) k_factor_lanes(int n, const int* __restrict__ rowPtr, const int* __restrict__ col,
                                                                const int* __restrict__ diag, const int* __restrict__ ford,
                                                                const int* __restrict__ elimPtr, const int* __restrict__ elimT,
                                                                const int* __restrict__ elimQ, const double* __restrict__ val, F* lu,
                                                                int* flagL, int epoch, unsigned* ctr, int* nreg, int* err) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        __syncwarp();
        const int base = warp_claim(ctr);
        if (base >= n) break;
        if (base + lane >= n) continue;
        const int i = __ldg(ford + base + lane);
        const int r0 = __ldg(rowPtr + i), r1 = __ldg(rowPtr + i + 1), d = __ldg(diag + i);
        W row[kLaneRow * 9];
        for (int e = 0; e < 9 * (r1 - r0); ++e) row[e] = W(F(__ldg(val + size_t(r0) * 9 + e)));
        for (int p0 = r0; p0 < d; p0 += 4) {                  // wait for the rows before it (bounded), four polled together
            int k[4];
            unsigned pending = 0, ns = 0;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                k[v] = p0 + v < d ? __ldg(col + p0 + v) : -1;
                if (k[v] >= 0) pending |= 1u << v;
            }
            for (unsigned it = 0; pending; ++it) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (((pending >> v) & 1u) && ld_relaxed(flagL + k[v]) == epoch) pending &= ~(1u << v);
                if (!pending || !poll_again(it, ns, err)) break;
            }
        }
        fence_acquire();
        for (int p = r0; p < d; ++p) {
            const int k = __ldg(col + p), q0 = __ldg(elimPtr + p), q1 = __ldg(elimPtr + p + 1);
            const F* u = lu + size_t(__ldg(diag + k)) * 9;
            W U[9], L[9];
            W* a = row + size_t(p - r0) * 9;
#pragma unroll
            for (int e = 0; e < 9; ++e) U[e] = W(u[e]);
#pragma unroll
            for (int e = 0; e < 9; ++e) {                     // L_ik = A_ik U_kk^-1
                W l = W(0);
#pragma unroll
                for (int m = 0; m < 3; ++m) l = fadd(l, fmul(a[3 * (e / 3) + m], U[3 * m + e % 3]));
                L[e] = l;
            }
#pragma unroll
            for (int e = 0; e < 9; ++e) a[e] = L[e];
            for (int q = q0; q < q1; ++q) {                   // A_it -= L_ik U_kq
                const F* f = lu + size_t(__ldg(elimQ + q)) * 9;
                W* t = row + size_t(__ldg(elimT + q) - r0) * 9;
#pragma unroll
                for (int e = 0; e < 9; ++e) U[e] = W(f[e]);
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    W s = W(0);
#pragma unroll
                    for (int m = 0; m < 3; ++m) s = fadd(s, fmul(L[3 * (e / 3) + m], U[3 * m + e % 3]));
                    t[e] = fsub(t[e], s);
                }
            }
        }
        double B[9];
        W* D = row + size_t(d - r0) * 9;
#pragma unroll
        for (int e = 0; e < 9; ++e) B[e] = double(D[e]);
        if (invert_pivot3(B)) atomicAdd(nreg, 1);
#pragma unroll
        for (int e = 0; e < 9; ++e) D[e] = W(B[e]);
        for (int e = 0; e < 9 * (r1 - r0); ++e) lu[size_t(r0) * 9 + e] = F(row[e]);
        st_release(flagL + i, epoch);
    }
}

// ------------------------------------------------------------------ sweeps
// Input modes of the forward sweep (fusions of the BiCGSTAB vector updates, engine/src/linsolve.cpp:172-186):
enum { IN_PLAIN = 0, IN_PUPDATE = 1, IN_SUPDATE = 2 };

__device__ __forceinline__ bool sys_running(const KScal* ks, const int* rowSys, int i) {
    return ks == nullptr || ks[__ldg(rowSys + i)].status == ST_RUNNING;
}

// Grid-wide BILU0 sweeps (engine/src/bsr.cpp:568-587). What bounds them is the chain of levels: a row's step is the trip of
// its neighbours' values through L2 and its own arithmetic. So:
// * the results travel as words that are their own flags (rsg_sync.cuh): a dependency costs one trip, with no flag, fence
//   or second load. Two word vectors: yf takes the forward results, yb the backward ones; each sweep clears the other's
//   words of its rows. Rows of systems that are not running are left out of both;
// * three lanes take a row, one component each, ten rows per claim: a third of a row's loads and FP64 operations per lane
//   (a warp of 32 rows kept the FP64 pipe of its SM busy for 0.4 us of every level);
// * everything that does not depend on a neighbour (factor blocks, the inverted diagonal, the input) is loaded before the
//   wait.
// TF: factor storage, TV: vector and arithmetic -- (double, double), (float, double): FP64 explicitly rounded, the
// reference's sweeps; (float, float): BILU0f (engine/src/bsr.cpp:1100-1121).
// IN_PUPDATE: in = p = r + beta (p - omega v) (p stored); IN_SUPDATE: in = s = r - alpha v (s stored in pv)

// yi -= sum_p (row e of B_p) . y_col(p) over the entries [p0, p1) of a row, in order, four entries at a time
template <class TF, class TV>
__device__ __forceinline__ void sub_polled(TV& yi, const int* __restrict__ col, const TF* __restrict__ lu, int p0, int p1, int e,
                                           const typename Word<TV>::type* y, int* err) {
    for (int q = p0; q < p1; q += 4) {
        int k[4];
        TF a[4][3];
        TV w[4][3];
        unsigned pending = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            k[u] = q + u < p1 ? __ldg(col + q + u) : -1;
            if (k[u] >= 0) pending |= 7u << (3 * u);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int f = 0; f < 3; ++f) a[u][f] = k[u] >= 0 ? __ldg(lu + size_t(q + u) * 9 + 3 * e + f) : TF(0);
        unsigned ns = 0;
        for (unsigned it = 0; pending; ++it) {
            typename Word<TV>::type got[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if ((pending >> (3 * u + f)) & 1u) got[u][f] = ld_word(y + size_t(k[u]) * 3 + f);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (((pending >> (3 * u + f)) & 1u) && got[u][f] != Word<TV>::empty) {
                        w[u][f] = Word<TV>::value(got[u][f]);
                        pending &= ~(1u << (3 * u + f));
                    }
            if (!pending || !poll_again(it, ns, err)) break;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (k[u] < 0) break;
            yi = vsub(yi, rdot(a[u], w[u]));
        }
    }
}

template <class TF, class TV, class TI, int MODE>
__global__ void __launch_bounds__(kSweepThreads) k_fwd(int n, const int* __restrict__ rowPtr, const int* __restrict__ col,
                                                       const int* __restrict__ diag, const int* __restrict__ ford, const TF* __restrict__ lu,
                                                       const TI* r, double* pv, const double* v, typename Word<TV>::type* yf,
                                                       typename Word<TV>::type* yb, const int* __restrict__ rowSys, const KScal* ks,
                                                       unsigned* ctr, int* err) {
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[1] = 0u;   // backward claim counter for the next sweep
    const int lane = threadIdx.x & 31, rr = lane / 3, e = lane % 3;
    for (;;) {
        __syncwarp();
        const int base = warp_claim(ctr, kSweepRows);
        if (base >= n) break;
        const int idx = base + rr;
        if (rr >= kSweepRows || idx >= n) continue;
        const int i = __ldg(ford + idx);
        if (!sys_running(ks, rowSys, i)) continue;
        const size_t q = size_t(i) * 3 + e;
        TV yi;
        if constexpr (MODE == IN_PLAIN) {
            yi = TV(r[q]);
        } else {
            const KScal& K = ks[__ldg(rowSys + i)];
            const double in = MODE == IN_PUPDATE ? da(r[q], dm(K.beta, ds(pv[q], dm(K.omega, v[q])))) : ds(r[q], dm(K.alpha, v[q]));
            pv[q] = in;
            yi = TV(in);
        }
        sub_polled<TF, TV>(yi, col, lu, __ldg(rowPtr + i), __ldg(diag + i), e, yf, err);
        st_word(yf + q, Word<TV>::make(yi));
        yb[q] = Word<TV>::empty;
    }
}

// The same for one long row by the whole warp (the cliques of perforated cells): 32 entries at a time, a lane each, all polled
// together; the products go through `sh` (96 words of the warp) to lanes 0 .. 2, which subtract them in entry order. Four
// entries at a time such a row costs two trips through L2 per four entries after the neighbour it waited for, and the rows of a
// clique wait for one another: in the backward sweep that neighbour comes first. 277,000 rows with five 42-layer wells, FP32:
// 485 -> 412 us; 180,000 rows with 30-layer wells, FP64: 487 -> 406 us. The forward sweep waits for the last entry, has done the
// others by then, and is slower this way (288 -> 363 us).
constexpr int kLongRow = 8;                  // entries a row's own lanes take (two rounds)
template <class TF, class TV>
__device__ __forceinline__ TV sub_polled_warp(TV yi, const int* __restrict__ col, const TF* __restrict__ lu, int p0, int p1,
                                              const typename Word<TV>::type* y, TV* sh, int* err) {
    const int lane = threadIdx.x & 31;
    for (int q = p0; q < p1; q += 32) {
        const int n = min(32, p1 - q);
        if (lane < n) {
            const int k = __ldg(col + q + lane);
            TF a[9];
            TV w[3] = {TV(0), TV(0), TV(0)};
#pragma unroll
            for (int f = 0; f < 9; ++f) a[f] = __ldg(lu + size_t(q + lane) * 9 + f);
            unsigned ns = 0, pending = 7;
            for (unsigned it = 0; pending; ++it) {
                typename Word<TV>::type got[3];
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if ((pending >> f) & 1u) got[f] = ld_word(y + size_t(k) * 3 + f);
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    if (((pending >> f) & 1u) && got[f] != Word<TV>::empty) {
                        w[f] = Word<TV>::value(got[f]);
                        pending &= ~(1u << f);
                    }
                if (!pending || !poll_again(it, ns, err)) break;
            }
#pragma unroll
            for (int f = 0; f < 3; ++f) sh[3 * lane + f] = rdot(a + 3 * f, w);
        }
        __syncwarp();
        if (lane < 3)
#pragma unroll 4
            for (int u = 0; u < n; ++u) yi = vsub(yi, sh[3 * u + lane]);
        __syncwarp();
    }
    return yi;
}
// A claim's rows in order: runs of short rows, three lanes each, and single long rows by the warp (a row may wait for an
// earlier one of the same claim)
template <class Short, class Long>
__device__ __forceinline__ void claim_rows(int rr, bool have, int len, Short&& shortRow, Long&& longRow) {
    const unsigned longs = __ballot_sync(0xffffffffu, have && len > kLongRow);
    for (int s = 0;;) {
        const unsigned m = longs >> (3 * s);                 // (bits 0 .. 29: three lanes a row)
        const int L = m ? s + (__ffs(int(m)) - 1) / 3 : kSweepRows;
        if (have && rr >= s && rr < L) shortRow();
        if (L >= kSweepRows) break;
        __syncwarp();
        longRow(3 * L);
        s = L + 1;
    }
}

// z_i = U_ii^-1 (y_i - sum_{j>i} U_ij z_j)   (engine/src/bsr.cpp:577-587); xp (CPR): z_p += xp as z is written (bsr.cpp:1083)
template <class TF, class TV, class TX>
__global__ void __launch_bounds__(kSweepThreads) k_bwd(int n, const int* __restrict__ rowPtr, const int* __restrict__ col,
                                                       const int* __restrict__ diag, const int* __restrict__ bord, const TF* __restrict__ lu,
                                                       typename Word<TV>::type* yf, typename Word<TV>::type* yb, double* z,
                                                       const TX* __restrict__ xp, const int* __restrict__ rowSys, const KScal* ks,
                                                       unsigned* ctr, int* err) {
    __shared__ TV sh[kSweepThreads * 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[0] = 0u;
    const int lane = threadIdx.x & 31, rr = lane / 3, e = lane % 3;
    const unsigned mine = 7u << (3 * rr);                    // the row's lanes (a warp's rows may depend on each other)
    for (;;) {
        __syncwarp();
        const int base = warp_claim(ctr + 1, kSweepRows);
        if (base >= n) break;
        const int idx = base + rr;
        int i = 0, d = 0, p1 = 0;
        bool have = rr < kSweepRows && idx < n;
        if (have) {
            i = __ldg(bord + idx);
            d = __ldg(diag + i);
            p1 = __ldg(rowPtr + i + 1);
            have = sys_running(ks, rowSys, i);
        }
        claim_rows(rr, have, p1 - d - 1,
            [&] {
                const size_t q = size_t(i) * 3 + e;
                TF D[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) D[f] = __ldg(lu + size_t(d) * 9 + 3 * e + f);
                const double corr = xp && e == 0 ? double(__ldg(xp + i)) : 0.0;
                TV yi = Word<TV>::value(yf[q]);
                yf[q] = Word<TV>::empty;
                sub_polled<TF, TV>(yi, col, lu, d + 1, p1, e, yb, err);
                TV w[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) w[f] = __shfl_sync(mine, yi, 3 * rr + f);
                const TV t = rdot(D, w);
                st_word(yb + q, Word<TV>::make(t));
                z[q] = xp && e == 0 ? da(double(t), corr) : double(t);
            },
            [&](int src) {
                const int ii = __shfl_sync(0xffffffffu, i, src), dd = __shfl_sync(0xffffffffu, d, src), b = __shfl_sync(0xffffffffu, p1, src);
                const size_t q = size_t(ii) * 3 + lane;
                TF D[3] = {TF(0), TF(0), TF(0)};
                TV yi = TV(0);
                double corr = 0.0;
                if (lane < 3) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) D[f] = __ldg(lu + size_t(dd) * 9 + 3 * lane + f);
                    if (xp && lane == 0) corr = double(__ldg(xp + ii));
                    yi = Word<TV>::value(yf[q]);
                    yf[q] = Word<TV>::empty;
                }
                yi = sub_polled_warp<TF, TV>(yi, col, lu, dd + 1, b, yb, sh + (threadIdx.x >> 5) * 96, err);
                TV w[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) w[f] = __shfl_sync(0xffffffffu, yi, f);
                if (lane < 3) {
                    const TV t = rdot(D, w);
                    st_word(yb + q, Word<TV>::make(t));
                    z[q] = xp && lane == 0 ? da(double(t), corr) : double(t);
                }
            });
    }
}

// ------------------------------------------------------------------ tile kernels with fused reductions (rsg_reduce.cuh)
// SpMV epilogues / fused dot products
enum { SP_PLAIN = 0, SP_RV = 1, SP_OMEGA = 2, SP_TRUERES = 3 };

// y = A x on one tile (3 threads per block row). SP_RV: partial <rh, y>; then alpha = rho / <rh, v>. SP_OMEGA:
// partials <t,t>, <t,s>, <s,s>; then omega or the early exit on ||s||. SP_TRUERES: y = b - A x, partials <y,y>,
// <b,b>, result sqrt ratio into out[s].
//
// Arithmetic (FMA): false = the reference's order and rounding per block (engine/src/bsr.cpp:109-117: row sum of
// the block from zero, then added; bitwise the reference), true = one fused multiply-add per term.
// On GB300 the FP64 unit runs at 1/64 of the FP32 rate, and the 9 multiply-adds of a block bound this kernel
// rather than HBM: the FMA form keeps the FP64 pipe about 90 % busy at 70 % of the HBM copy rate, the unfused
// form needs twice the FP64 instructions. Hence direct read-only loads (the values stream once, the x gather
// hits L2), 128 block rows per pass so the SM holds enough loads in flight, and a reduction that spends as few
// FP64 adds as possible (rsg_reduce.cuh).
constexpr int kSpmvThreads = 384;

template <bool FMA>
__device__ __forceinline__ double block_row_term(double yv, const double* a, const double* xc) {
    if (FMA) return fma(a[2], __ldg(xc + 2), fma(a[1], __ldg(xc + 1), fma(a[0], __ldg(xc), yv)));
    return da(yv, da(da(dm(a[0], __ldg(xc)), dm(a[1], __ldg(xc + 1))), dm(a[2], __ldg(xc + 2))));
}

template <int MODE>
__device__ __forceinline__ void spmv_out(size_t q, double yv, double* y, const double* __restrict__ a1, double (&acc)[MAX_DOTS]) {
    if (MODE == SP_TRUERES) {
        const double bq = __ldg(a1 + q);
        const double rq = ds(bq, yv);
        if (y) y[q] = rq;
        acc[0] += rq * rq;
        acc[1] += bq * bq;
    } else {
        y[q] = yv;
        if (MODE == SP_RV) acc[0] += __ldg(a1 + q) * yv;
        if (MODE == SP_OMEGA) {
            const double sq = __ldg(a1 + q);
            acc[0] += yv * yv;
            acc[1] += yv * sq;
            acc[2] += sq * sq;
        }
    }
}

template <int MODE, bool FMA>
__global__ void __launch_bounds__(kSpmvThreads) k_spmv_tile(int ntiles, int nsys, const int* __restrict__ tileRow0,
                                                           const int* __restrict__ tileSys, const int* __restrict__ sysTile0,
                                                           const int* __restrict__ rowPtr, const int* __restrict__ col,
                                                           const double* __restrict__ val, const double* __restrict__ x, double* y,
                                                           const double* __restrict__ a1, KScal* ks, double* part, unsigned* done,
                                                           double* sysdot, int* active, double* out) {
    __shared__ double sh[MAX_DOTS * kSpmvThreads];
    const int tile = blockIdx.x;
    const int s = __ldg(tileSys + tile);
    const bool run = (MODE == SP_PLAIN || MODE == SP_TRUERES) || ks[s].status == ST_RUNNING;
    double acc[MAX_DOTS] = {0, 0, 0, 0};
    if (run) {
        const int r0 = __ldg(tileRow0 + tile), r1 = __ldg(tileRow0 + tile + 1);
        const int e = threadIdx.x % 3;
        for (int row = r0 + int(threadIdx.x) / 3; row < r1; row += kSpmvThreads / 3) {
            double yv = 0;
            const int p1 = __ldg(rowPtr + row + 1);
            for (int p = __ldg(rowPtr + row); p < p1; ++p) {
                const double* a = val + size_t(p) * 9 + e * 3;
                const double av[3] = {__ldg(a), __ldg(a + 1), __ldg(a + 2)};
                yv = block_row_term<FMA>(yv, av, x + size_t(__ldg(col + p)) * 3);
            }
            spmv_out<MODE>(size_t(row) * 3 + e, yv, y, a1, acc);
        }
    }
    if (MODE == SP_PLAIN) return;
    constexpr int ND = MODE == SP_RV ? 1 : (MODE == SP_OMEGA ? 3 : 2);
    block_reduce<ND>(acc, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int j = 0; j < ND; ++j) part[size_t(tile) * MAX_DOTS + j] = acc[j];
    if (!last_tile_reduce<ND>(ntiles, nsys, sysTile0, part, done, sysdot, sh)) return;
    for (int q = threadIdx.x; q < nsys; q += blockDim.x) {
        const double* dd = sysdot + size_t(q) * MAX_DOTS;
        if (MODE == SP_TRUERES) {
            out[q] = dd[1] > 0 ? sqrt(dd[0]) / sqrt(dd[1]) : 0.0;
            continue;
        }
        KScal& K = ks[q];
        if (K.status != ST_RUNNING) continue;
        if (MODE == SP_RV) {
            const double rv = dd[0];
            if (fabs(rv) < 1e-300 || !isfinite(rv)) {   // engine/src/linsolve.cpp:179
                K.status = ST_BREAKDOWN;
                atomicSub(active, 1);
            } else {
                K.alpha = K.rho / rv;
            }
        } else if (MODE == SP_OMEGA) {
            const double tt = dd[0], ts = dd[1], ss = dd[2];
            K.sn = sqrt(ss);
            K.omega = tt > 0 ? ts / tt : 0.0;             // engine/src/linsolve.cpp:196
        }
    }
}

// BiCGSTAB initial state: x = 0, r = rh = b, p = v = 0; rho = <b,b>, alpha = omega = 1 (engine/src/linsolve.cpp:162-168)
__global__ void __launch_bounds__(kTileThreads) k_bicg_init(int ntiles, int nsys, const int* __restrict__ tileRow0,
                                                           const int* __restrict__ tileSys, const int* __restrict__ sysTile0,
                                                           const double* __restrict__ b, double* x, double* r, double* rh, double* p,
                                                           double* v, KScal* ks, double tol, int maxit, int guard, int onlyFailed,
                                                           double* part, unsigned* done, double* sysdot, int* active) {
    __shared__ double sh[MAX_DOTS * kTileThreads];
    const int tile = blockIdx.x;
    const size_t q0 = size_t(__ldg(tileRow0 + tile)) * 3, q1 = size_t(__ldg(tileRow0 + tile + 1)) * 3;
    double acc[MAX_DOTS] = {0, 0, 0, 0};
    // onlyFailed: the systems that converged keep their solution and status (a restart of the others)
    if (!onlyFailed || ks[__ldg(tileSys + tile)].status != ST_CONV)
        for (size_t q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
            const double bq = __ldg(b + q);
            x[q] = 0; r[q] = bq; rh[q] = bq; p[q] = 0; v[q] = 0;
            acc[0] += bq * bq;
        }
    block_reduce<1>(acc, sh);
    if (threadIdx.x == 0) part[size_t(tile) * MAX_DOTS] = acc[0];
    if (!last_tile_reduce<1>(ntiles, nsys, sysTile0, part, done, sysdot, sh)) return;
    if (threadIdx.x == 0) *active = 0;
    __syncthreads();
    int nact = 0;
    for (int s = threadIdx.x; s < nsys; s += blockDim.x) {
        KScal& K = ks[s];
        if (onlyFailed && K.status == ST_CONV) continue;
        const double bb = sysdot[size_t(s) * MAX_DOTS];
        K.guard = guard;
        K.hn = 1e300;           // the guard's best residual so far and its iteration
        K.gj = 0;
        K.bn = sqrt(bb);
        K.tol = tol; K.maxit = maxit; K.its = 0; K.relres = 0; K.sn = 0;
        K.alpha = 1; K.omega = 1; K.rho = bb; K.beta = bb;   // rhoN of iteration 1 = <rh, r> = <b, b>
        if (K.bn == 0) { K.status = ST_CONV; }                // engine/src/linsolve.cpp:165
        else if (fabs(bb) < 1e-300 || !isfinite(bb)) { K.status = ST_BREAKDOWN; }
        else if (maxit < 1) { K.status = ST_MAXIT; }
        else { K.status = ST_RUNNING; ++nact; }
    }
    if (nact) atomicAdd(active, nact);
}

// End of a BiCGSTAB iteration (engine/src/linsolve.cpp:183-213):
//   ||s|| small: x += alpha ph and stop; else x += alpha ph + omega sh, r = s - omega t, then ||r||, <rh, r>.
__global__ void __launch_bounds__(kTileThreads) k_bicg_update(int ntiles, int nsys, const int* __restrict__ tileRow0,
                                                             const int* __restrict__ tileSys, const int* __restrict__ sysTile0,
                                                             double* x, double* r, const double* __restrict__ rh,
                                                             const double* __restrict__ s, const double* __restrict__ t,
                                                             const double* __restrict__ ph, const double* __restrict__ sh_,
                                                             KScal* ks, double* part, unsigned* done, double* sysdot, int* active) {
    __shared__ double sh[MAX_DOTS * kTileThreads];
    const int tile = blockIdx.x;
    const int sy = __ldg(tileSys + tile);
    KScal K = ks[sy];
    double acc[MAX_DOTS] = {0, 0, 0, 0};
    if (K.status == ST_RUNNING) {
        const size_t q0 = size_t(__ldg(tileRow0 + tile)) * 3, q1 = size_t(__ldg(tileRow0 + tile + 1)) * 3;
        const bool sconv = K.sn / K.bn < K.tol;
        for (size_t q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
            if (sconv) {
                x[q] = da(x[q], dm(K.alpha, __ldg(ph + q)));
            } else {
                x[q] = da(x[q], da(dm(K.alpha, __ldg(ph + q)), dm(K.omega, __ldg(sh_ + q))));
                const double rq = ds(__ldg(s + q), dm(K.omega, __ldg(t + q)));
                r[q] = rq;
                acc[0] += rq * rq;
                acc[1] += __ldg(rh + q) * rq;
            }
        }
    }
    block_reduce<2>(acc, sh);
    if (threadIdx.x == 0) { part[size_t(tile) * MAX_DOTS] = acc[0]; part[size_t(tile) * MAX_DOTS + 1] = acc[1]; }
    if (!last_tile_reduce<2>(ntiles, nsys, sysTile0, part, done, sysdot, sh)) return;
    for (int q = threadIdx.x; q < nsys; q += blockDim.x) {
        KScal& k = ks[q];
        if (k.status != ST_RUNNING) continue;
        const int it = k.its + 1;
        k.its = it;
        if (k.sn / k.bn < k.tol) {                              // engine/src/linsolve.cpp:187-191
            k.relres = k.sn / k.bn;
            k.status = ST_CONV;
            atomicSub(active, 1);
            continue;
        }
        const double rn = sqrt(sysdot[size_t(q) * MAX_DOTS]);
        const double rhoN = sysdot[size_t(q) * MAX_DOTS + 1];
        k.relres = rn / k.bn;
        if (rn / k.bn < k.tol) { k.status = ST_CONV; atomicSub(active, 1); continue; }
        if (k.omega == 0 || !isfinite(rn)) { k.status = ST_BREAKDOWN; atomicSub(active, 1); continue; }
        if (fabs(rhoN) < 1e-300) { k.status = ST_BREAKDOWN; atomicSub(active, 1); continue; }   // next iteration's test
        if (it >= k.maxit) { k.status = ST_MAXIT; atomicSub(active, 1); continue; }
        if (k.guard) {          // FP32 preconditioner: diverging, or no new best residual for 40 iterations (stalled)
            if (k.relres < k.hn) { k.hn = k.relres; k.gj = it; }
            if ((it >= 8 && k.relres > 1e4) || it - k.gj >= 40) { k.status = ST_DIVERGED; atomicSub(active, 1); continue; }
        }
        k.beta = (rhoN / k.rho) * (k.alpha / k.omega);
        k.rho = rhoN;
    }
}

// ------------------------------------------------------------------ block Jacobi
__global__ void k_bj_setup(int n, const int* __restrict__ diag, const double* __restrict__ val, double* dinv, int* nreg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double D[9];
    load9_ro(val + size_t(__ldg(diag + i)) * 9, D);
    double B[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) B[e] = D[e];
    if (!invert3(B)) {   // DeviceCprAmg fallback: 1 / max(1e-30, |D_ee|) (engine/src/bsr.cpp:1305)
#pragma unroll
        for (int e = 0; e < 9; ++e) B[e] = 0;
        for (int e = 0; e < 3; ++e) B[e * 4] = 1.0 / fmax(1e-30, fabs(D[e * 4]));
        atomicAdd(nreg, 1);
    }
    store9(dinv + size_t(i) * 9, B);
}

template <int MODE>
__global__ void k_bj_apply(int n, const double* __restrict__ dinv, const double* r, double* pv, const double* v, double* z,
                           const int* __restrict__ rowSys, const KScal* ks) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool run = sys_running(ks, rowSys, i);
    if (!run) return;
    double yi[3];
    if (MODE == IN_PUPDATE) {
        const KScal& K = ks[__ldg(rowSys + i)];
        for (int e = 0; e < 3; ++e) {
            const size_t q = size_t(i) * 3 + e;
            const double pe = da(r[q], dm(K.beta, ds(pv[q], dm(K.omega, v[q]))));
            pv[q] = pe; yi[e] = pe;
        }
    } else if (MODE == IN_SUPDATE) {
        const KScal& K = ks[__ldg(rowSys + i)];
        for (int e = 0; e < 3; ++e) {
            const size_t q = size_t(i) * 3 + e;
            const double se = ds(r[q], dm(K.alpha, v[q]));
            pv[q] = se; yi[e] = se;
        }
    } else {
        for (int e = 0; e < 3; ++e) yi[e] = r[size_t(i) * 3 + e];
    }
    double D[9];
    load9_ro(dinv + size_t(i) * 9, D);
    z[size_t(i) * 3 + 0] = dot3(D, yi);
    z[size_t(i) * 3 + 1] = dot3(D + 3, yi);
    z[size_t(i) * 3 + 2] = dot3(D + 6, yi);
}

__global__ void k_gather_blocks(int nnzb, const int* __restrict__ src, const double* __restrict__ a, double* b) {
    const size_t total = size_t(nnzb) * 9;
    for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < total; q += size_t(gridDim.x) * blockDim.x)
        b[q] = __ldg(a + size_t(__ldg(src + q / 9)) * 9 + q % 9);
}
// Four words a thread and round, their loads issued together: a word is two dependent loads (742,384 rows: gather 9.9 -> 9.4 us,
// scatter 9-10 us either way; a product with both 121.7 -> 120.4 us; 40 MB, 6 us of HBM time). A vector that the grid covers in
// one round takes a word a thread (80,000 rows: a product 24.6 us, with four 25.8).
template <bool GATHER, int U>
__device__ __forceinline__ void permute_vec(int n, const int* __restrict__ perm, const double* __restrict__ from, double* to) {
    const size_t total = size_t(n) * 3, step = size_t(gridDim.x) * blockDim.x;
    for (size_t q0 = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q0 < total; q0 += U * step) {
        size_t at[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t q = q0 + u * step;
            const unsigned row = q < total ? unsigned(q / 3) : 0u;
            at[u] = size_t(__ldg(perm + row)) * 3 + size_t(q - size_t(row) * 3);
            if (!GATHER && q < total) v[u] = __ldg(from + q);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (GATHER && q0 + u * step < total) v[u] = __ldg(from + at[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t q = q0 + u * step;
            if (q < total) to[GATHER ? q : at[u]] = v[u];
        }
    }
}
template <int U>
__global__ void __launch_bounds__(256) k_gather_vec(int n, const int* __restrict__ perm, const double* __restrict__ orig, double* lev) {
    permute_vec<true, U>(n, perm, orig, lev);
}
template <int U>
__global__ void __launch_bounds__(256) k_scatter_vec(int n, const int* __restrict__ perm, const double* __restrict__ lev, double* orig) {
    permute_vec<false, U>(n, perm, lev, orig);
}

int g_sm_count = 0;
int stream_grid(size_t total) {
    const size_t g = (total + 255) / 256, cap = size_t(device_sm_count()) * 16;
    return int(g < cap ? (g > 0 ? g : 1) : cap);
}
}  // namespace

// Persistent grid of a sync-free pass whose warps claim rowsPerWarp rows each: `inflight` levels of avgRows rows in flight (a
// warp far ahead of the front only polls), at most 8 blocks of 4 warps per SM, which is what auto takes. CPR application, grid-wide,
// auto / 32 / 8 / 2 levels: 180,000 rows FP64 3.85 / 3.75 / 3.77 / 4.24 ms, 277,000 rows FP32 1.26 / 1.28 / 1.53 / 2.73 ms, 11,200 rows
// FP64 1.24 / 1.22 / 1.26 / 1.28 ms; factorisation 4.9, 13.5 and 2.07 ms, the same from two levels on.
int sweep_blocks_for(double avgRows, int inflight, int rowsPerWarp) {
    const long long cap = 8LL * device_sm_count();
    if (inflight <= 0) return int(cap);
    const double warps = double(inflight) * avgRows / double(rowsPerWarp);
    const long long blocks = (long long)((warps + 3.0) / 4.0);
    return int(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

int device_sm_count() {
    if (g_sm_count == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (g_sm_count <= 0) g_sm_count = 1;
    }
    return g_sm_count;
}

void launch_gather_blocks(const DevPlan& P, const double* src, double* dst, cudaStream_t st) {
    k_gather_blocks<<<stream_grid(size_t(P.nnzb) * 9), 256, 0, st>>>(P.nnzb, P.valSrc, src, dst);
}
void launch_gather_vec(const DevPlan& P, const double* orig, double* lev, cudaStream_t st) {
    const int g = stream_grid(size_t(P.n) * 3);
    if (size_t(g) * 256 >= size_t(P.n) * 3) k_gather_vec<1><<<g, 256, 0, st>>>(P.n, P.perm, orig, lev);
    else k_gather_vec<4><<<g, 256, 0, st>>>(P.n, P.perm, orig, lev);
}
void launch_scatter_vec(const DevPlan& P, const double* lev, double* orig, cudaStream_t st) {
    const int g = stream_grid(size_t(P.n) * 3);
    if (size_t(g) * 256 >= size_t(P.n) * 3) k_scatter_vec<1><<<g, 256, 0, st>>>(P.n, P.perm, lev, orig);
    else k_scatter_vec<4><<<g, 256, 0, st>>>(P.n, P.perm, lev, orig);
}

// a row per warp in a persistent grid; several rows per claim only where a level (of the whole batch) has more rows than the
// grid has warps
template <class W, class F>
static void launch_factor_t(const DevPlan& P, const double* val, F* lu, W* work, SweepState& S, int epoch, int* nreg, int* err,
                            cudaStream_t st) {
    cudaMemsetAsync(S.ctr + 2, 0, sizeof(unsigned), st);
    if (P.maxRowBlocks <= kLaneRow && P.avgLevelRows >= (sizeof(W) == 8 ? 70.0 : 30.0) * device_sm_count()) {
        const int g = std::max(1, std::min(8 * device_sm_count(), (P.n + kSweepThreads - 1) / kSweepThreads));
        k_factor_lanes<W, F><<<g, kSweepThreads, 0, st>>>(P.n, P.rowPtr, P.col, P.diag, P.ford, P.elimPtr, P.elimT, P.elimQ, val, lu, S.flagL, epoch,
                                                         S.ctr + 2, nreg, err);
        return;
    }
    const int blocks = std::max(1, std::min(P.factorBlocks, (P.n + 3) / 4));
    const int chunk = std::max(1, std::min(8, int(P.avgLevelRows / double(blocks * (kSweepThreads / 32)))));
    k_factor<W, F><<<blocks, kSweepThreads, 0, st>>>(P.n, chunk, P.rowPtr, P.col, P.diag, P.ford, P.elimPtr, P.elimT, P.elimQ, val, lu, work,
                                                    S.flagL, epoch, S.ctr + 2, nreg, err);
}
void launch_factor_f64(const DevPlan& P, const double* val, double* lu, SweepState& S, int epoch, int* nreg, int* err,
                       cudaStream_t st) {
    launch_factor_t<double, double>(P, val, lu, lu, S, epoch, nreg, err, st);
}
void launch_factor_lean(const DevPlan& P, const double* val, float* luf, double* work, SweepState& S, int epoch, int* nreg,
                        int* err, cudaStream_t st) {
    launch_factor_t<double, float>(P, val, luf, work, S, epoch, nreg, err, st);
}
void launch_factor_f32(const DevPlan& P, const double* val, float* luf, SweepState& S, int epoch, int* nreg, int* err, cudaStream_t st) {
    launch_factor_t<float, float>(P, val, luf, luf, S, epoch, nreg, err, st);
}

// both sweeps, the input by mode
template <class TF, class TV, class TI, class TX>
static void launch_sweeps(const DevPlan& P, const TF* lu, int mode, const TI* r, double* pv, const double* v, double* z, const TX* xp,
                          const KScal* ks, SweepState& S, int* err, cudaStream_t st) {
    using U = typename Word<TV>::type;
    const int g = std::min(P.sweepBlocks, std::max(1, (P.n + 4 * kSweepRows - 1) / (4 * kSweepRows)));
    U* yf = reinterpret_cast<U*>(S.yw);
    U* yb = reinterpret_cast<U*>(S.yw + size_t(P.n) * 3);
    auto fwd = [&](auto tag) {
        k_fwd<TF, TV, TI, decltype(tag)::value><<<g, kSweepThreads, 0, st>>>(P.n, P.rowPtr, P.col, P.diag, P.ford, lu, r, pv, v, yf, yb, P.rowSys,
                                                                             ks, S.ctr, err);
    };
    if (mode == IN_PLAIN) fwd(std::integral_constant<int, IN_PLAIN>());
    else if constexpr (sizeof(TI) == 8) {
        if (mode == IN_PUPDATE) fwd(std::integral_constant<int, IN_PUPDATE>());
        else fwd(std::integral_constant<int, IN_SUPDATE>());
    }
    k_bwd<TF, TV, TX><<<g, kSweepThreads, 0, st>>>(P.n, P.rowPtr, P.col, P.diag, P.bord, lu, yf, yb, z, xp, P.rowSys, ks, S.ctr, err);
}
void launch_ilu_grid(const DevPlan& P, const PrecDev& M, int mode, const double* r, double* pv, const double* v, double* z, const KScal* ks,
                     SweepState& S, int* err, cudaStream_t st) {
    const double* no = nullptr;
    if (M.kind == 0) launch_sweeps<double, double>(P, M.lu, mode, r, pv, v, z, no, ks, S, err, st);
    else if (M.kind == 1) launch_sweeps<float, double>(P, M.luf, mode, r, pv, v, z, no, ks, S, err, st);
    else launch_sweeps<float, float>(P, M.luf, mode, r, pv, v, z, no, ks, S, err, st);
}
// second stage of a CPR application: t in FP64, or (split form of the all-FP32 preconditioner) in FP32; z_p += xp
void launch_ilu_grid_cpr(const DevPlan& P, const PrecDev& M, const double* t, const float* tf, const DevAmg& G, double* z, const KScal* ks,
                         SweepState& S, int* err, cudaStream_t st) {
    if (M.kind == 0) launch_sweeps<double, double>(P, M.lu, IN_PLAIN, t, nullptr, nullptr, z, G.x, ks, S, err, st);
    else if (M.kind == 1) launch_sweeps<float, double>(P, M.luf, IN_PLAIN, t, nullptr, nullptr, z, G.xf, ks, S, err, st);
    else if (tf) launch_sweeps<float, float>(P, M.luf, IN_PLAIN, tf, nullptr, nullptr, z, G.xf, ks, S, err, st);
    else launch_sweeps<float, float>(P, M.luf, IN_PLAIN, t, nullptr, nullptr, z, G.xf, ks, S, err, st);
}

template <int MODE, bool FMA>
void spmv_go(const DevPlan& P, const double* val, const double* x, double* y, const double* a1, KScal* ks, ReduceState* R, int* active,
             double* out, cudaStream_t st) {
    k_spmv_tile<MODE, FMA><<<P.ntiles, kSpmvThreads, 0, st>>>(P.ntiles, P.nsys, P.tileRow0, P.tileSys, P.sysTile0, P.rowPtr, P.col, val,
                                                               x, y, a1, ks, R ? R->part : nullptr, R ? R->done : nullptr,
                                                               R ? R->sysdot : nullptr, active, out);
}
// SpMV tile kernel with the handle's arithmetic (P.spmvFma)
template <int MODE>
void spmv(const DevPlan& P, const double* val, const double* x, double* y, const double* a1, KScal* ks, ReduceState* R, int* active,
          double* out, cudaStream_t st) {
    if (P.spmvFma) spmv_go<MODE, true>(P, val, x, y, a1, ks, R, active, out, st);
    else spmv_go<MODE, false>(P, val, x, y, a1, ks, R, active, out, st);
}

// The dynamic shared-memory opt-in of a kernel is one process-wide value per device: handles on several threads
// (serving slots) with plans of different sizes only ever raise it, under one lock. Without it a launch may have 48 KB of
// static and dynamic shared memory together (the static part of every kernel here is below 32 KB).
void raise_smem_limit(const void* fn, int bytes) {
    if (bytes <= 16 * 1024) return;
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> lim;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto [it, first] = lim.try_emplace({dev, fn}, 0);
    if (first) {
        cudaFuncAttributes a{};
        if (cudaFuncGetAttributes(&a, fn) == cudaSuccess) it->second = std::max(0, 48 * 1024 - int(a.sharedSizeBytes));
    }
    if (bytes > it->second) {
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        it->second = bytes;
    }
}

__global__ void k_vec_add(size_t m, double* x, const double* __restrict__ d) {
    for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < m; q += size_t(gridDim.x) * blockDim.x) x[q] += d[q];
}
void launch_vec_add(int n, double* x, const double* d, cudaStream_t st) {
    const size_t m = size_t(n) * 3;
    const int g = int(std::min<size_t>((m + 255) / 256, size_t(device_sm_count()) * 8));
    k_vec_add<<<std::max(g, 1), 256, 0, st>>>(m, x, d);
}

void launch_spmv_f64(const DevPlan& P, const double* val, const double* x, double* y, cudaStream_t st) {
    spmv<SP_PLAIN>(P, val, x, y, nullptr, nullptr, nullptr, nullptr, nullptr, st);
}

void launch_block_jacobi_setup(const DevPlan& P, const double* val, double* dinv, int* nreg, cudaStream_t st) {
    k_bj_setup<<<(P.n + 127) / 128, 128, 0, st>>>(P.n, P.diag, val, dinv, nreg);
}
void launch_block_jacobi_apply(const DevPlan& P, const double* dinv, const double* r, double* z, cudaStream_t st) {
    k_bj_apply<IN_PLAIN><<<(P.n + 127) / 128, 128, 0, st>>>(P.n, dinv, r, nullptr, nullptr, z, P.rowSys, nullptr);
}

void launch_bicg_init(const DevPlan& P, const double* b, BicgVecs& V, KScal* ks, ReduceState& R, double tol, int maxit,
                      int* active, bool guard, bool onlyFailed, cudaStream_t st) {
    k_bicg_init<<<P.ntiles, kTileThreads, 0, st>>>(P.ntiles, P.nsys, P.tileRow0, P.tileSys, P.sysTile0, b, V.x, V.r, V.rh, V.p, V.v,
                                                   ks, tol, maxit, guard ? 1 : 0, onlyFailed ? 1 : 0, R.part, R.done, R.sysdot, active);
}

// one iteration: (a) p-update fused into M p, (c) v = A ph + <rh,v>, (d) s-update fused into M s,
// (f) t = A sh + <t,t>, <t,s>, <s,s>, (g) x / r update + ||r||, <rh,r>
void launch_bicg_iteration(const DevPlan& P, const double* val, const PrecDev& M, BicgVecs& V, KScal* ks, ReduceState& R,
                           SweepState& S, int* active, int* err, cudaStream_t st) {
    auto prec = [&](bool pupd, double* out) {
        if (M.devcpr) {
            launch_devcpr(P, *M.amg, val, pupd ? 1 : 2, V.r, pupd ? V.p : V.s, V.v, out, ks, st);
        } else if (M.cpr && M.cta && !M.split) {
            launch_cpr_cta(P, M, *M.amg, pupd ? 1 : 2, M.kind != 0, V.r, pupd ? V.p : V.s, V.v, out, ks, st);
        } else if (M.cpr) {
            launch_cpr_grid(P, M, *M.amg, pupd ? 1 : 2, V.r, pupd ? V.p : V.s, V.v, out, ks, S, err, st);
        } else if (M.cta && M.kind != 2) {
            launch_ilu_cta_fused(P, M, pupd, V.r, pupd ? V.p : V.s, V.v, out, ks, st);
        } else if (M.kind != 2) {
            launch_ilu_grid(P, M, pupd ? IN_PUPDATE : IN_SUPDATE, V.r, pupd ? V.p : V.s, V.v, out, ks, S, err, st);
        } else {
            const int gb = (P.n + 127) / 128;
            if (pupd)
                k_bj_apply<IN_PUPDATE><<<gb, 128, 0, st>>>(P.n, M.dinv, V.r, V.p, V.v, out, P.rowSys, ks);
            else
                k_bj_apply<IN_SUPDATE><<<gb, 128, 0, st>>>(P.n, M.dinv, V.r, V.s, V.v, out, P.rowSys, ks);
        }
    };
    prec(true, V.ph);
    spmv<SP_RV>(P, val, V.ph, V.v, V.rh, ks, &R, active, nullptr, st);
    prec(false, V.sh);
    spmv<SP_OMEGA>(P, val, V.sh, V.t, V.s, ks, &R, active, nullptr, st);
    k_bicg_update<<<P.ntiles, kTileThreads, 0, st>>>(P.ntiles, P.nsys, P.tileRow0, P.tileSys, P.sysTile0, V.x, V.r, V.rh, V.s, V.t,
                                                     V.ph, V.sh, ks, R.part, R.done, R.sysdot, active);
}

void launch_true_residual(const DevPlan& P, const double* val, const double* b, const double* x, double* tmp, ReduceState& R,
                          double* out, cudaStream_t st) {
    spmv<SP_TRUERES>(P, val, x, tmp, b, nullptr, &R, nullptr, out, st);
}

}  // namespace rsg
