// BILU0 sweeps of one system per thread block, fed by a shared-memory ring of bulk copies.
//
// The sweeps of BILU0::apply (engine/src/bsr.cpp:437-596) are a chain of dependent levels (forward levels of L, then the
// same levels in reverse for U: structurally symmetric patterns). A level step is short, so what bounds the chain is what
// a step waits for besides its own arithmetic. Here:
// * the sweep vector of the system lives in shared memory for both sweeps (the input is copied in, the forward result
//   stays, the backward sweep overwrites it), so a step gathers its neighbours from shared memory;
// * a producer warp brings every level's factor records (row-major: a thread reads its row with 16-byte loads free of
//   bank conflicts), slot columns, overflow blocks and CPR corrections into a byte ring by bulk copies
//   (cp.async.bulk), as many levels ahead as the ring holds; a level's rows are contiguous in level space, so a level is
//   four copies. Neither the consumers' registers nor the level barriers carry loads from L2;
// * a consumer holds two rows in registers: while it waits for its neighbours' values of one step it reads the record of
//   its row of the next one, so a step is barrier, gather, arithmetic, store;
// * two writer warps store the results of the previous step (z_p += xp, the conversion to FP64, which runs on the slow
//   FP64 pipe), off the chain.
// FP64 vectors take three lanes per row (one component each): the FP64 pipe (2 lanes per SM per clock) is the bound
// there, and a third of the dependent operations per lane shortens the step. FP32 takes one thread per row.
//
// Measured against the sweeps with register lookahead and per-thread staging (rsg_sweep_cta.cu), both sweeps of one
// application: all FP32, 11,200 rows alone 178 -> 113 us, 1,600 rows 84 -> 43 us, 64 systems of 8,000-14,400 rows
// 250 -> 157 us (the largest vector leaves the ring 50 KB: one to two steps ahead); FP64, 1,600 rows 232 -> 127 us. What is
// left of a step (0.6 us at 130 rows) is the shared-memory traffic of its records, written once and read once, and the
// barrier. FP64 vectors of more than about 6,000 rows do not fit and stay with the other sweeps.
//
// Arithmetic: the reference's order per row (slots, then the overflow list, in row order), FP64 unfused, as the sweeps of
// rsg_sweep_cta.cu; the results are the same bit for bit.
#include "rsg_impl.h"
#include "rsg_block3.cuh"
#include "rsg_ring.cuh"

#include <cuda_runtime.h>
#include <type_traits>

namespace rsg {

namespace {

constexpr int kRingWriters = 64;           // writer threads; beside them the consumers and one producer warp
constexpr int kRingFlight = 16;            // steps in flight at most (mbarriers of the ring)
constexpr uint32_t kRingHeader = kRingFlight * 32 + 16;   // full and empty mbarriers, step infos, input mbarrier (+ pad)
// steps between a step's prefetch into L2 and its copy: where the vector leaves the ring room for one wide step only, a copy's
// latency is on the chain (64 systems of 8,000-14,400 rows, 187 MB of factors an application: 169 -> 157 us)
constexpr int kRingPrefetch = 6;
constexpr size_t kRingReserve = 1024;      // shared memory the runtime keeps per block
// rows of one step at most (a wider level is several steps): one per consumer thread (FP32), or ten per warp (FP64)
// (FP32 steps of 128 rows would let two fit a short ring: 157 -> 168 us, alone 99 -> 115 us, by the added barriers)
constexpr int kRingRows32 = 256, kRingRows64 = 120;
template <class TV> __host__ __device__ constexpr int ring_rows() { return sizeof(TV) == 8 ? kRingRows64 : kRingRows32; }
template <class TV> __host__ __device__ constexpr int ring_max_threads() { return (sizeof(TV) == 8 ? 384 : 256) + kRingWriters + 32; }

template <class TF> __host__ __device__ constexpr uint32_t ov_words() { return sizeof(TF) == 4 ? 12 : 10; }   // block, column, pad

template <class TF>
struct RingArgs {
    const int* sysRow0;
    const int* stepOff;                    // per system: its steps are desc[stepOff[s] .. stepOff[s + 1])
    const int4* desc;                      // per step: {first row, rows | overflow entries << 16, first overflow entry, 0}
    const int4 *Lslot, *Uslot;
    const TF *L, *UD, *Lov, *Uov;          // row-major records; overflow entries {9 values, column, pad}
};

template <class TF>
__device__ __forceinline__ int ov_col(const TF* e) {
    if constexpr (sizeof(TF) == 4) return __float_as_int(e[9]);
    else return __double2loint(e[9]);
}

// a row of a step in registers: slot columns, factor values (one thread per row: three blocks and, backward, the inverted
// diagonal; three lanes per row: one block row of each)
template <class TF, int LPR>
struct RingRow {
    int k, ov;                             // row (system; -1: none), offset of the step's overflow entries in the ring
    bool held;                             // the step has overflow lists: its ring bytes are read until its end
    int4 c;
    TF a[LPR == 3 ? 9 : 28], D[LPR == 3 ? 3 : 9];
};
template <class TF>
__device__ __forceinline__ void ring_row_load(RingRow<TF, 3>& R, const TF* rec, const int4* slots, int t, int e, bool fwd) {
    R.c = slots[t];
    const TF* p = rec + size_t(t) * (fwd ? LREC : UREC) + 3 * e;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int f = 0; f < 3; ++f) R.a[3 * j + f] = p[9 * j + f];
    if (!fwd) {
#pragma unroll
        for (int f = 0; f < 3; ++f) R.D[f] = p[27 + f];
    }
}
__device__ __forceinline__ void ring_row_load(RingRow<float, 1>& R, const float* rec, const int4* slots, int t, int, bool fwd) {
    R.c = slots[t];
    const float4* p = reinterpret_cast<const float4*>(rec + size_t(t) * (fwd ? LREC : UREC));
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        const float4 q = p[j];
        R.a[4 * j] = q.x; R.a[4 * j + 1] = q.y; R.a[4 * j + 2] = q.z; R.a[4 * j + 3] = q.w;
    }
    if (!fwd) {
        const float4 q = p[7], w = p[8];
        R.D[0] = R.a[27]; R.D[1] = q.x; R.D[2] = q.y; R.D[3] = q.z; R.D[4] = q.w; R.D[5] = w.x; R.D[6] = w.y; R.D[7] = w.z; R.D[8] = w.w;
    }
}

// IN: 0 the input is a TV vector (copied in), 1 a double vector, 2 the p-update, 3 the s-update of BiCGSTAB (stored to pv).
// XP: the CPR pressure correction xp is added to z_p as z is written.
template <class TF, class TV, int IN, bool XP, class TX>
__global__ void __launch_bounds__(ring_max_threads<TV>(), 1) k_ring(RingArgs<TF> A, const TV* T, const double* r, double* pv, const double* v,
                                                                 double* z, const TX* x, const AmgSysLv* __restrict__ lv, int maxL,
                                                                 const KScal* ks, uint32_t smemBytes, int* err) {
    constexpr int LPR = sizeof(TV) == 8 ? 3 : 1;             // lanes per row
    constexpr int RPW = LPR == 3 ? 10 : 32;                  // rows per warp
    extern __shared__ __align__(16) unsigned char sm[];
    const int s = blockIdx.x, tid = int(threadIdx.x), nc = int(blockDim.x) - kRingWriters - 32;
    double beta = 0, omega = 0, alpha = 0;
    if (ks) {
        const KScal& K = ks[s];
        if (K.status != ST_RUNNING) return;                  // whole block: uniform
        beta = K.beta; omega = K.omega; alpha = K.alpha;
    }
    const int row0 = __ldg(A.sysRow0 + s), ns = __ldg(A.sysRow0 + s + 1) - row0;
    const int d0 = __ldg(A.stepOff + s), S = __ldg(A.stepOff + s + 1) - d0, nl = S / 2;
    const int x0 = XP ? __ldg(&lv[s * maxL].rowOff) : 0;
    // a step in the ring: {record offset, slot column offset, first row (system) << 10 | has overflow entries << 9 | rows,
    // offset of its first overflow entry}
    int4* info = reinterpret_cast<int4*>(sm + kRingFlight * 16);
    int4* desc = reinterpret_cast<int4*>(sm + kRingHeader);
    // the vector, placed so that it is as far from a 16-byte boundary as its input in global memory (bulk copy)
    const size_t inByte = size_t(row0) * 3 * sizeof(TV);
    unsigned char* ybase = sm + kRingHeader + size_t(S) * sizeof(int4);
    TV* y = reinterpret_cast<TV*>(ybase + (IN == 0 ? (inByte & 15) : 0));
    const uint32_t yBytes = (uint32_t(ns) * 3 * sizeof(TV) + 31) & ~15u;
    unsigned char* ring = ybase + yBytes;
    const uint32_t full = smem_addr(sm), empty = full + kRingFlight * 8, inBar = full + kRingFlight * 32, ringA = smem_addr(ring);
    for (int i = tid; i < S; i += int(blockDim.x)) desc[i] = __ldg(A.desc + d0 + i);
    if (tid == 0) {
        for (int i = 0; i < kRingFlight; ++i) {
            mbar_init(full + 8 * i, 1);
            mbar_init(empty + 8 * i, uint32_t(nc + kRingWriters) / 32);
        }
        mbar_init(inBar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int dead = 0;                                            // 1 + the step whose wait ran out
    const int lane = tid & 31;
    auto step_end = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nc + kRingWriters) : "memory"); };
    auto await = [&](int step) { mbar_wait(full + 8 * (step % kRingFlight), (step / kRingFlight) & 1, dead, err, step + 1); };
    if (tid >= nc + kRingWriters) {                          // ---- producer: one thread
        if (lane) return;
        if (IN == 0) {                                       // the 16-byte aligned middle of the input
            const uint32_t bytes = uint32_t(ns) * 3 * sizeof(TV), mid0 = uint32_t((16 - (inByte & 15)) & 15);
            const uint32_t mid = bytes > mid0 ? (bytes - mid0) & ~15u : 0;
            mbar_expect_tx(inBar, mid);
            if (mid) bulk_load(smem_addr(y) + mid0, reinterpret_cast<const unsigned char*>(T) + inByte + mid0, mid, inBar);
        }
        ByteRing R{smemBytes - uint32_t(ring - sm)};
        int oldest = 0;                                      // steps oldest .. next - 1 hold ring bytes
        auto prefetch = [&](int step) {
            if (step >= S) return;
            const int4 d = desc[step];
            const bool f = step < nl;
            const uint32_t n = uint32_t(d.y) & 0xffffu;
            bulk_prefetch((f ? A.L : A.UD) + size_t(d.x) * (f ? LREC : UREC), n * uint32_t((f ? LREC : UREC) * sizeof(TF)));
            bulk_prefetch((f ? A.Lslot : A.Uslot) + d.x, 16 * n);
        };
        for (int step = 1; step < kRingPrefetch; ++step) prefetch(step);
        for (int next = 0; next < S; ++next) {
            prefetch(next + kRingPrefetch);
            const int4 d = desc[next];
            const bool f = next < nl;
            const uint32_t n = uint32_t(d.y) & 0xffffu;
            const uint32_t rec = n * uint32_t((f ? LREC : UREC) * sizeof(TF)), ov = (uint32_t(d.y) >> 16) * uint32_t(ov_words<TF>() * sizeof(TF));
            uint32_t xp = 0;                                 // backward: a 16-byte aligned window around the step's corrections
            uint64_t xa = 0;
            if (XP && !f) {
                xa = reinterpret_cast<uint64_t>(x) + uint64_t(x0 + d.x - row0) * sizeof(TX);
                xp = (uint32_t(xa & 15) + n * uint32_t(sizeof(TX)) + 15) & ~15u;
                xa &= ~15ull;
            }
            const uint32_t bytes = rec + 16 * n + xp + ov;
            uint32_t at = 0;
            while (next - oldest >= kRingFlight || !R.alloc(bytes, at)) {
                mbar_wait(empty + 8 * (oldest % kRingFlight), (oldest / kRingFlight) & 1, dead, err);
                if (dead) return;                            // (the steps not issued are skipped by whoever waits for them)
                ++oldest;
                R.free_oldest(oldest < next ? uint32_t(info[oldest % kRingFlight].x) : 0);
            }
            info[next % kRingFlight] = make_int4(int(at), int(at + rec), ((d.x - row0) << 10) | (ov ? 512 : 0) | int(n),
                                                 int(at + rec + 16 * n + xp));
            const uint32_t bar = full + 8 * (next % kRingFlight);
            mbar_expect_tx(bar, bytes);
            uint32_t dst = ringA + at;
            bulk_load(dst, (f ? A.L : A.UD) + size_t(d.x) * (f ? LREC : UREC), rec, bar);
            dst += rec;
            bulk_load(dst, (f ? A.Lslot : A.Uslot) + d.x, 16 * n, bar);
            dst += 16 * n;
            if (xp) bulk_load(dst, reinterpret_cast<const void*>(xa), xp, bar);
            if (ov) bulk_load(dst + xp, (f ? A.Lov : A.Uov) + size_t(d.z) * ov_words<TF>(), ov, bar);
        }
        return;
    }
    if (tid >= nc) {                                         // ---- writers
        const int w = tid - nc;
        constexpr int RPT = (ring_rows<TV>() + kRingWriters - 1) / kRingWriters;
        int n = 0, k0 = 0;                                   // the step before: its rows and corrections
        TX xp[RPT];
        auto store = [&]() {
#pragma unroll
            for (int q = 0; q < RPT; ++q) {
                const int t = w + q * kRingWriters;
                if (t >= n) break;
                const TV* yk = y + 3 * (k0 + t);
                double* zk = z + size_t(row0 + k0 + t) * 3;
                zk[0] = XP ? da(double(yk[0]), double(xp[q])) : double(yk[0]);
                zk[1] = double(yk[1]);
                zk[2] = double(yk[2]);
            }
        };
        for (int step = 0; step <= S; ++step) {
            int4 d = make_int4(0, 0, 0, 0);
            TX xn[RPT];
            if (step >= nl && step < S) {
                await(step);
                if (!dead) d = info[step % kRingFlight];
                if (XP) {
                    const uint64_t xa = reinterpret_cast<uint64_t>(x) + uint64_t(x0 + (d.z >> 10)) * sizeof(TX);
                    const TX* xs = reinterpret_cast<const TX*>(ring + d.y + 16 * (d.z & 511) + (xa & 15));
#pragma unroll
                    for (int q = 0; q < RPT; ++q) xn[q] = w + q * kRingWriters < (d.z & 511) ? xs[w + q * kRingWriters] : TX(0);
                }
            }
            __syncwarp();
            if (lane == 0 && step < S) mbar_arrive(empty + 8 * (step % kRingFlight));
            step_end();                                      // the step before is final
            store();
            n = d.z & 511;
            k0 = d.z >> 10;
            if (XP) {
#pragma unroll
                for (int q = 0; q < RPT; ++q) xp[q] = xn[q];
            }
        }
        return;
    }
    // ---- consumers: the input
    if (IN == 0) {
        const uint32_t bytes = uint32_t(ns) * 3 * sizeof(TV), m0 = uint32_t((16 - (inByte & 15)) & 15);
        const uint32_t e0 = min(uint32_t(ns) * 3, m0 / uint32_t(sizeof(TV)));
        const uint32_t e1 = bytes > m0 ? (m0 + ((bytes - m0) & ~15u)) / uint32_t(sizeof(TV)) : e0;
        for (uint32_t i = tid; i < e0; i += nc) y[i] = T[size_t(row0) * 3 + i];
        for (uint32_t i = e1 + tid; i < uint32_t(ns) * 3; i += nc) y[i] = T[size_t(row0) * 3 + i];
        mbar_wait(inBar, 0, dead, err);
    } else {
        constexpr int U = 8;
        for (int base = tid; base < 3 * ns; base += U * nc) {
            double a[U], b[U], c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const size_t q = size_t(row0) * 3 + size_t(min(base + u * nc, 3 * ns - 1));
                a[u] = r[q];
                b[u] = IN == 2 ? pv[q] : 0.0;
                c[u] = IN >= 2 ? v[q] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = base + u * nc;
                if (i >= 3 * ns) break;
                double in = a[u];
                if (IN == 2) in = da(a[u], dm(beta, ds(b[u], dm(omega, c[u]))));   // linsolve.cpp:173
                if (IN == 3) in = ds(a[u], dm(alpha, c[u]));                       // linsolve.cpp:183
                if (IN >= 2) pv[size_t(row0) * 3 + i] = in;
                y[i] = TV(in);
            }
        }
    }
    // ---- consumers: the steps
    const int rw = LPR == 3 ? lane / 3 : lane, e = LPR == 3 ? lane % 3 : 0, t0 = (tid >> 5) * RPW + rw;
    const bool mine = LPR == 1 || lane < 30;
    using Row = RingRow<TF, LPR>;
    int gate = lane;                                         // 0: gives the warp's bytes back
    auto fetch = [&](Row& R, int step) {
        await(step);
        int4 d = info[step % kRingFlight];
        // After a wait that ran out `info` may be another step's: no rows, and whether the step has lists (which decides the warp
        // synchronisations that follow) from the step table, as the other lanes see it. The bytes are not given back then:
        // the producer would reuse them under a copy. (Checks outside this branch -- a vote, `&& !dead` at the arrivals, the
        // producer waiting for the copies -- cost 0.5 to 2 % of a sweep.)
        if (dead) {
            gate = 32;
            d.z = uint32_t(desc[step].y) >> 16 ? 512 : 0;
        }
        R.k = mine && t0 < (d.z & 511) ? (d.z >> 10) + t0 : -1;
        R.ov = d.w;
        R.c.w = -1;
        if (R.k >= 0)
            ring_row_load(R, reinterpret_cast<const TF*>(ring + d.x), reinterpret_cast<const int4*>(ring + d.y), t0, e, step < nl);
        R.held = (d.z & 512) != 0;
        __syncwarp();                                        // (the arrival releases the reads of all lanes, not of lane 0 alone)
        if (!R.held && gate == 0) mbar_arrive(empty + 8 * (step % kRingFlight));
    };
    auto body = [&](Row& R, Row& N, int step) {
        const bool fwd = step < nl;
        constexpr int NO = LPR == 3 ? 1 : 3;
        TV yi[NO], yc[9];
        step_end();
        if (R.k >= 0) {                                      // gather: every load issued before any is used
#pragma unroll
            for (int f = 0; f < NO; ++f) yi[f] = y[3 * R.k + (LPR == 3 ? e : f)];
#pragma unroll
            for (int j = 0; j < SLOTS; ++j) {
                const int cj = j == 0 ? R.c.x : (j == 1 ? R.c.y : R.c.z), cs = cj >= 0 ? cj : R.k;   // (an empty slot reads a value it drops)
#pragma unroll
                for (int f = 0; f < 3; ++f) yc[3 * j + f] = y[3 * cs + f];
            }
        }
        // a warp that still holds ring bytes of this step does not wait for the next one before it has released them (the
        // ring need not have room for both)
        const bool held = R.held;
        if (!held && step + 1 < S) fetch(N, step + 1);
        if (R.k >= 0) {
#pragma unroll
            for (int j = 0; j < SLOTS; ++j) {
                const int cj = j == 0 ? R.c.x : (j == 1 ? R.c.y : R.c.z);
#pragma unroll
                for (int f = 0; f < NO; ++f) {
                    const TV u = vsub(yi[f], rdot(R.a + (LPR == 3 ? 3 * j : 9 * j + 3 * f), yc + 3 * j));
                    yi[f] = cj >= 0 ? u : yi[f];
                }
            }
            if (R.c.w >= 0) {
                constexpr int OW = int(ov_words<TF>());
                const uint32_t at = ring_entry(uint32_t(R.ov), R.c.w, desc[step].z, uint32_t(OW * sizeof(TF)));
                for (const TF* o = reinterpret_cast<const TF*>(ring + at);; o += OW) {
                    const int cj = ov_col(o);
                    if (cj < 0) break;
                    const TV w[3] = {y[3 * cj], y[3 * cj + 1], y[3 * cj + 2]};
#pragma unroll
                    for (int f = 0; f < NO; ++f) yi[f] = vsub(yi[f], rdot(o + (LPR == 3 ? 3 * e : 3 * f), w));
                }
            }
        }
        if constexpr (LPR == 3) {
            if (!fwd) {                                      // the row's three components from its lanes
                TV w[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) w[f] = __shfl_sync(0xffffffffu, yi[0], lane - e + f);
                yi[0] = rdot(R.D, w);
            }
            if (R.k >= 0) y[3 * R.k + e] = yi[0];
        } else if (R.k >= 0) {
            TV w[3] = {yi[0], yi[1], yi[2]};
            if (!fwd) {
#pragma unroll
                for (int f = 0; f < 3; ++f) w[f] = rdot(R.D + 3 * f, yi);
            }
#pragma unroll
            for (int f = 0; f < 3; ++f) y[3 * R.k + f] = w[f];
        }
        if (held) {
            __syncwarp();
            if (gate == 0) mbar_arrive(empty + 8 * (step % kRingFlight));
            if (step + 1 < S) fetch(N, step + 1);
        }
    };
    Row P, Q;
    fetch(P, 0);
    for (int step = 0; step < S; step += 2) {
        body(P, Q, step);
        if (step + 1 < S) body(Q, P, step + 1);
    }
    step_end();                                              // (the writers store the last step)
    if (dead) {                                              // the block ends after the copies in flight have landed (in order, to the first not issued)
        int late = 0;
        if (IN == 0) mbar_wait(inBar, 0, late, err);
        for (int step = dead - 1; step < S && !late; ++step) mbar_wait(full + 8 * (step % kRingFlight), (step / kRingFlight) & 1, late, err);
    }
}

// factors (level-space CSR block order) -> row-major slot records and overflow entries
template <class T>
__global__ void k_ring_pack(int n, int nLov, int nUov, const int* __restrict__ LslotSrc, const int* __restrict__ UslotSrc,
                            const int* __restrict__ Dsrc, const int* __restrict__ LovSrc, const int* __restrict__ UovSrc,
                            const int* __restrict__ LovCol, const int* __restrict__ UovCol, const T* __restrict__ lu, T* L, T* UD, T* Lov,
                            T* Uov) {
    constexpr size_t OW = ov_words<T>();
    const size_t nL = size_t(n) * LREC, nUD = size_t(n) * UREC, nO = (size_t(nLov) + size_t(nUov)) * OW;
    for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < nL + nUD + nO; q += size_t(gridDim.x) * blockDim.x) {
        if (q < nL) {
            const size_t k = q / LREC, e = q % LREC, j = e / 9;
            const int src = j < size_t(SLOTS) ? __ldg(LslotSrc + k * SLOTS + j) : -1;
            L[q] = src >= 0 ? lu[size_t(src) * 9 + e % 9] : T(0);
        } else if (q < nL + nUD) {
            const size_t q2 = q - nL, k = q2 / UREC, e = q2 % UREC, j = e / 9;
            const int src = j < size_t(SLOTS) ? __ldg(UslotSrc + k * SLOTS + j) : __ldg(Dsrc + k);
            UD[q2] = src >= 0 ? lu[size_t(src) * 9 + e % 9] : T(0);
        } else {
            const size_t q3 = q - nL - nUD, b = q3 / OW, e = q3 % OW;
            const bool lo = b < size_t(nLov);
            const size_t i = lo ? b : b - size_t(nLov);
            const int src = __ldg((lo ? LovSrc : UovSrc) + i), col = __ldg((lo ? LovCol : UovCol) + i);
            T val = T(0);
            if (e < 9) val = src >= 0 ? lu[size_t(src) * 9 + e] : T(0);
            else if (e == 9) {
                if constexpr (sizeof(T) == 4) val = __int_as_float(col);
                else val = __hiloint2double(0, col);
            }
            (lo ? Lov : Uov)[i * OW + e] = val;
        }
    }
}

size_t smem_cap() {
    static int v = 0;
    if (!v) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (v <= 0) v = 48 * 1024;
    }
    return size_t(v) - kRingReserve;
}

// shared memory of a launch: the largest system's steps and vector, and a ring of as much as is left, at most kRingWant and
// no more than all its steps take, so that blocks of small systems share an SM; with more systems than SMs also no more than
// lets two blocks share one. Both sweeps, 128 KB for every block / so: 1,000 systems of 100 rows FP64 203 / 103 us, FP32 96 / 51 us;
// 300 of 400 117 / 80 and 62 / 39 us; 300 of 1,600 FP32 121 / 68 us (four blocks: 69; 300 of 3,300: two 154, four 173 us).
// 0: the largest level of some system does not fit
constexpr size_t kRingWant = 128 * 1024;
constexpr int kRingShare = 2;
size_t ring_smem(const RingDev& R, size_t sizeTF, size_t sizeTV, int nsys) {
    const size_t fixed = kRingHeader + size_t(R.maxSteps) * sizeof(int4) + ((size_t(R.maxRows) * 3 * sizeTV + 31) & ~size_t(15));
    const size_t stage = (sizeTF == 4 ? R.maxStage32 : R.maxStage64) + 32;
    const size_t cap = smem_cap();
    if (R.maxSteps == 0 || fixed + stage > cap) return 0;
    size_t want = std::min(kRingWant, (sizeTF == 4 ? R.maxBytes32 : R.maxBytes64) + 32);
    if (nsys > device_sm_count()) {
        const size_t share = (cap + kRingReserve) / size_t(kRingShare) - kRingReserve;
        want = std::min(want, share > fixed ? share - fixed : 0);
    }
    return std::min(cap, fixed + std::max(stage, want));
}

template <class TF, class TV, int IN, bool XP, class TX>
void launch_ring_t(const DevPlan& P, const RingDev& R, const RingFactors<TF>& F, const TV* T, const double* r, double* pv, const double* v,
                   double* z, const TX* x, const AmgSysLv* lv, int maxL, const KScal* ks, int* err, cudaStream_t st) {
    const size_t sm = ring_smem(R, sizeof(TF), sizeof(TV), P.nsys);
    const auto fn = k_ring<TF, TV, IN, XP, TX>;
    raise_smem_limit(reinterpret_cast<const void*>(fn), int(sm));
    // a thread (FP64 vectors: three lanes of a warp's thirty) per row of the widest level, in whole warps
    const int rpw = sizeof(TV) == 8 ? 10 : 32;
    const int warps = std::max(1, (R.maxWidth + rpw - 1) / rpw);
    fn<<<P.nsys, 32 * warps + kRingWriters + 32, sm, st>>>(RingArgs<TF>{P.sysRow0, R.stepOff, R.desc, P.Lslot, P.Uslot, F.L, F.UD, F.Lov, F.Uov}, T, r, pv, v,
                                            z, x, lv, maxL, ks, uint32_t(sm), err);
}

}  // namespace

bool ring_fits(const RingDev& R, bool factors32, bool vec32) { return ring_smem(R, factors32 ? 4 : 8, vec32 ? 4 : 8, 1) > 0; }

void ring_steps(const HostPlan& P, bool vec32, RingHost& H) {
    const int kRows = vec32 ? kRingRows32 : kRingRows64;
    H = RingHost{};
    H.stepOff.assign(size_t(P.nsys) + 1, 0);
    for (int s = 0; s < P.nsys; ++s) {
        const int l0 = P.sysLvl0[size_t(s)], nl = P.sysLvl0[size_t(s) + 1] - l0 - 1;
        H.maxRows = std::max(H.maxRows, P.sysRow0[size_t(s) + 1] - P.sysRow0[size_t(s)]);
        std::vector<std::pair<int, int>> rows;               // a system's steps in forward order
        for (int l = 0; l < nl; ++l) {
            const int a = P.lvlStart[size_t(l0 + l)], b = P.lvlStart[size_t(l0 + l) + 1];
            for (int k = a; k < b; k += kRows) rows.push_back({k, std::min(b, k + kRows)});
        }
        const int ns = int(rows.size());
        size_t all32 = 0, all64 = 0;
        H.maxSteps = std::max(H.maxSteps, 2 * ns);
        for (int g = 0; g < 2 * ns; ++g) {
            const bool f = g < ns;
            const int a = rows[size_t(f ? g : 2 * ns - 1 - g)].first, b = rows[size_t(f ? g : 2 * ns - 1 - g)].second;
            const std::vector<int>& slot = f ? P.Lslot : P.Uslot;
            const std::vector<int>& oc = f ? P.LovCol : P.UovCol;
            int ov0 = 0, ov1 = 0;                            // the step's overflow lists are contiguous (lists in row order)
            for (int k = a; k < b; ++k) {
                const int q = slot[size_t(k) * 4 + 3];
                if (q < 0) continue;
                if (ov1 == 0) ov0 = q;
                ov1 = q;
                while (oc[size_t(ov1)] >= 0) ++ov1;
                ++ov1;                                       // the terminator
            }
            const size_t n = size_t(b - a), ov = size_t(ov1 - ov0);
            if (ov > 0xffff) return;
            H.maxWidth = std::max(H.maxWidth, b - a);
            const size_t stage32 = n * (size_t(f ? LREC : UREC) * 4 + 16 + 4) + 32 + ov * ov_words<float>() * 4;
            const size_t stage64 = n * (size_t(f ? LREC : UREC) * 8 + 16 + 8) + 32 + ov * ov_words<double>() * 8;
            H.maxStage32 = std::max(H.maxStage32, stage32);
            H.maxStage64 = std::max(H.maxStage64, stage64);
            all32 += stage32;
            all64 += stage64;
            H.desc.push_back(make_int4(a, int(n | (ov << 16)), ov0, 0));
        }
        H.maxBytes32 = std::max(H.maxBytes32, all32);
        H.maxBytes64 = std::max(H.maxBytes64, all64);
        H.stepOff[size_t(s) + 1] = int(H.desc.size());
    }
    H.ok = true;
}

template <class T>
static void pack_t(const DevPlan& P, const T* lu, RingFactors<T>& F, cudaStream_t st) {
    const size_t total = size_t(P.n) * (LREC + UREC) + (size_t(P.nLov) + size_t(P.nUov)) * ov_words<T>();
    const int grid = int(std::min<size_t>((total + 255) / 256, size_t(device_sm_count()) * 16));
    k_ring_pack<T><<<grid, 256, 0, st>>>(P.n, P.nLov, P.nUov, P.LslotSrc, P.UslotSrc, P.Dsrc, P.LovSrc, P.UovSrc, P.LovCol, P.UovCol, lu, F.L, F.UD,
                                         F.Lov, F.Uov);
}
void launch_ring_pack(const DevPlan& P, const double* lu, RingFactors<double>& F, cudaStream_t st) { pack_t(P, lu, F, st); }
void launch_ring_pack(const DevPlan& P, const float* luf, RingFactors<float>& F, cudaStream_t st) { pack_t(P, luf, F, st); }
size_t ring_ov_words(bool factors32) { return factors32 ? ov_words<float>() : ov_words<double>(); }

// z = M^-1 in, the input by mode (0 plain, 1 p-update, 2 s-update); systems whose status is not running skip
void launch_ring_ilu(const DevPlan& P, const PrecDev& M, int mode, const double* r, double* pv, const double* v, double* z, const KScal* ks,
                     int* err, cudaStream_t st) {
    const RingDev& R = M.ring[M.kind == 3 ? 1 : 0];
    auto go = [&](auto tag) {
        constexpr int IN = decltype(tag)::value;
        if (M.kind == 0) launch_ring_t<double, double, IN, false, double>(P, R, M.r64, nullptr, r, pv, v, z, nullptr, nullptr, 0, ks, err, st);
        else if (M.kind == 1) launch_ring_t<float, double, IN, false, float>(P, R, M.r32, nullptr, r, pv, v, z, nullptr, nullptr, 0, ks, err, st);
        else launch_ring_t<float, float, IN, false, float>(P, R, M.r32, nullptr, r, pv, v, z, nullptr, nullptr, 0, ks, err, st);
    };
    if (mode == 1) go(std::integral_constant<int, 2>());
    else if (mode == 2) go(std::integral_constant<int, 3>());
    else go(std::integral_constant<int, 1>());
}

// second stage of the split CPR application: T in the sweep vector's type, z_p += x (level 0 of every system)
void launch_ring_cpr2(const DevPlan& P, const PrecDev& M, const DevAmg& G, const void* T, double* z, const KScal* ks, int* err,
                      cudaStream_t st) {
    const RingDev& R = M.ring[M.kind == 3 ? 1 : 0];
    if (M.kind == 0)
        launch_ring_t<double, double, 0, true, double>(P, R, M.r64, static_cast<const double*>(T), nullptr, nullptr, nullptr, z, G.x, G.lv, G.maxL, ks,
                                                       err, st);
    else if (M.kind == 1)
        launch_ring_t<float, double, 0, true, float>(P, R, M.r32, static_cast<const double*>(T), nullptr, nullptr, nullptr, z, G.xf, G.lv, G.maxL, ks,
                                                     err, st);
    else
        launch_ring_t<float, float, 0, true, float>(P, R, M.r32, static_cast<const float*>(T), nullptr, nullptr, nullptr, z, G.xf, G.lv, G.maxL, ks, err,
                                                    st);
}

}  // namespace rsg
