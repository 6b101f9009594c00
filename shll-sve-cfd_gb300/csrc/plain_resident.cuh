// Plain 1D runs with several time steps per launch (temporal blocking): the reference's arithmetic of
// shll_plain.cuh, cell by cell the same operations as the one-launch-per-step kernel k_step1, so the
// results are the same bits.
//
// A chunk of consecutive cells belongs to one block, which computes a window of its own cells and
// ORDER * S cells on each side, one thread per cell; S steps use up the window's margin, so that only
// every S steps (a sweep) the blocks exchange cells through L2.  What bounds a run of a small or
// middle-sized tube is the chain of one step (FP64: 2 divisions, a square root and about 14 dependent
// FP64 instructions of 64 clocks, some 2000 clocks; float about 500) and, for larger ones, the FP64
// pipe (19 clocks per warp instruction per SM): one chunk per SM gives every step the least of both,
// and the launch, its gap and the exchange are paid once per sweep.
//
// Resident form (chunks <= SMs): one cooperative launch runs all sweeps; a block waits (bounded) only
// for the progress counters of the chunks its window reaches.  Otherwise one launch per sweep.
#pragma once
#include <cmath>

#include "shll_plain.cuh"

namespace SHLL_PLAIN_NS {

constexpr int kResThreads = 512;             // most threads of a block (the window's cells)
constexpr long kResSpin = 1L << 20;          // polls before a block gives up (under a second)

__device__ __forceinline__ unsigned res_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

template <typename REAL>
struct ResArgs {
    REAL* U[2];        // state planes: sweep q reads U[q & 1] and writes U[(q + 1) & 1]
    int n;             // cells (and plane stride)
    int S;             // steps per sweep
    long steps;        // steps of the run
    unsigned* prog;    // sweeps completed per chunk, kPlainProgStride apart (resident form), else null
    int* flag;
    int stall;         // test hook: this chunk never publishes its progress (-1: none)
};

// LANES: threads per cell, 1, or 4 (FP64): lane q of a cell's group holds component q (lane 3 doubles
// component 0 and stores nothing)
template <typename REAL, int ORDER>
constexpr size_t res_smem(int cells) {
    return (size_t)(ORDER == 1 ? 12 : 18) * cells * sizeof(REAL);
}

template <typename REAL, int ORDER, int LANES>
__global__ void __launch_bounds__(kResThreads, 1) k_resident1(ResArgs<REAL> A, Gas<REAL> g) {
    extern __shared__ __align__(16) unsigned char res_raw[];
    constexpr int NQ = LANES == 1 ? 3 : 1;               // components of this thread
    const int T = blockDim.x / LANES, tid = threadIdx.x / LANES, n = A.n;   // window cells, this thread's
    const int lane = LANES == 1 ? 0 : threadIdx.x & 3;
    const int q0 = lane == 3 ? 0 : lane;                 // first component
    const bool writes = LANES == 1 || lane < 3;
    REAL* flux = reinterpret_cast<REAL*>(res_raw);     // [2][fp, fm][3][T], by step parity
    REAL* slp = flux + 12 * T;                         // order 2: [dp, dm][3][T]
    const long k = gridDim.x, c = blockIdx.x;
    const int a = (int)(c * n / k), b = (int)((c + 1) * n / k);   // own cells
    const int H = ORDER * A.S;
    const int i = a - H + tid;                         // this thread's cell
    const bool own = i >= a && i < b;
    // the chunks that own the window's cells (cell x belongs to chunk ((x + 1) k - 1) / n)
    const int first = max(a - H, 0), last = min(b + H, n) - 1;
    const int c0 = (int)(((first + 1) * k - 1) / n), nc = (int)(((last + 1) * k - 1) / n) - c0 + 1;
    REAL u[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) u[q] = q0 + q == 1 ? (REAL)0 : (REAL)1;
    int bad = 0, par = 0;
    for (long sweep = 0; sweep * A.S < A.steps; sweep++) {
        const int s_now = (int)min((long)A.S, A.steps - sweep * A.S);
        const REAL* Uin = (sweep & 1) ? A.U[1] : A.U[0];
        REAL* Uout = (sweep & 1) ? A.U[0] : A.U[1];
        if (sweep > 0) {
            // every chunk of the window has completed the previous sweep: its cells can be read, and
            // it no longer reads the buffer that this sweep writes
            bool ok = true;
            for (int q = threadIdx.x; q < nc; q += blockDim.x) {
                const unsigned* p = A.prog + (long)(c0 + q) * kPlainProgStride;
                bool got = c0 + q == c;
                for (long it = 0; it < kResSpin && !got; it++) {
                    got = res_acquire(p) >= (unsigned)sweep;
                    if (!got) {
                        if ((it & 63) == 63 && (res_acquire(reinterpret_cast<const unsigned*>(A.flag)) & SHLL_FLAG_TIMEOUT))
                            break;   // another block gave up
                        __nanosleep(20);
                    }
                }
                if (!got) atomicOr(A.flag, SHLL_FLAG_TIMEOUT);
                ok = ok && got;
            }
            if (!__syncthreads_and(ok)) return;
        }
        // cells valid before step s: [a - ORDER (s_now - s), b + ORDER (s_now - s)) within the tube
        if (i >= max(a - ORDER * s_now, 0) && i < min(b + ORDER * s_now, n) && (sweep == 0 || !own)) {
#pragma unroll
            for (int q = 0; q < NQ; q++) u[q] = __ldcg(Uin + (long)(q0 + q) * n + i);
        }
        for (int s = 0; s < s_now; s++, par ^= 1) {
            const int lo = a - ORDER * (s_now - s), hi = b + ORDER * (s_now - s);
            const bool valid = i >= max(lo, 0) && i < min(hi, n);
            const bool next = i >= max(lo + ORDER, 0) && i < min(hi - ORDER, n);
            REAL* F = flux + par * 6 * T;
            REAL fp[NQ], fm[NQ];
            if constexpr (LANES == 1) {
                if (valid) bad |= cell1(g, u, fp, fm);
            } else {
                // (whole warps, as the lanes of a group exchange their values)
                if (__any_sync(0xffffffffu, valid)) {
                    const int b = cell1_lanes(g, u[0], fp[0], fm[0]);
                    bad |= valid && b;
                }
            }
            if (valid && writes) {
#pragma unroll
                for (int q = 0; q < NQ; q++) { F[(q0 + q) * T + tid] = fp[q]; F[(3 + q0 + q) * T + tid] = fm[q]; }
            }
            __syncthreads();
            if constexpr (ORDER == 1) {
                if (next) {
                    REAL x[NQ], v[NQ];
                    bool special = false;
#pragma unroll
                    for (int q = 0; q < NQ; q++) {
                        // reflective walls (base_shll.c:93-110)
                        const REAL sg = (q0 + q == 1) ? (REAL)1 : (REAL)-1;
                        const REAL L = i == 0 ? sg * fm[q] : F[(q0 + q) * T + tid - 1];
                        const REAL Rr = i == n - 1 && i != 0 ? sg * fp[q] : F[(3 + q0 + q) * T + tid + 1];
                        x[q] = fp[q] - fm[q] + Rr - L;
                        v[q] = sub_scaled_plain(u[q], g.sx, x[q], &special);
                    }
#pragma unroll
                    for (int q = 0; q < NQ; q++) u[q] = special ? sub_scaled(u[q], g.sx, x[q]) : v[q];
                }
            } else {
                REAL dp[NQ], dm[NQ];
#pragma unroll
                for (int q = 0; q < NQ; q++) dp[q] = dm[q] = 0;
                if (valid && i >= max(lo + 1, 0) && i < min(hi - 1, n)) {
                    if (i > 0 && i < n - 1) {
                        bool special = false;
#pragma unroll
                        for (int q = 0; q < NQ; q++) {
                            dp[q] = slope_plain(g, F[(q0 + q) * T + tid - 1], fp[q], F[(q0 + q) * T + tid + 1], &special);
                            dm[q] = slope_plain(g, F[(3 + q0 + q) * T + tid - 1], fm[q], F[(3 + q0 + q) * T + tid + 1], &special);
                        }
                        if (special) {
#pragma unroll
                            for (int q = 0; q < NQ; q++) {
                                dp[q] = slope(g, F[(q0 + q) * T + tid - 1], fp[q], F[(q0 + q) * T + tid + 1]);
                                dm[q] = slope(g, F[(3 + q0 + q) * T + tid - 1], fm[q], F[(3 + q0 + q) * T + tid + 1]);
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < NQ; q++) if (writes) { slp[(q0 + q) * T + tid] = dp[q]; slp[(3 + q0 + q) * T + tid] = dm[q]; }
                }
                __syncthreads();
                if (next) {   // outflow walls (2nd_order_base_shll.c:210-262)
                    REAL x[NQ], y[NQ], v[NQ];
                    bool special = false;
#pragma unroll
                    for (int q = 0; q < NQ; q++) {
                        const bool wl = i == 0, wr = i == n - 1 && i != 0;
                        const REAL L = wl ? fp[q] : F[(q0 + q) * T + tid - 1], Ldf = wl ? (REAL)0 : slp[(q0 + q) * T + tid - 1];
                        const REAL Rr = wr ? fm[q] : F[(3 + q0 + q) * T + tid + 1];
                        const REAL Rdf = wr ? (REAL)0 : slp[(3 + q0 + q) * T + tid + 1];
                        x[q] = fp[q] - fm[q] + Rr - L;
                        y[q] = dp[q] + dm[q] - Rdf - Ldf;
                        v[q] = sub_half_scaled_plain(sub_scaled_plain(u[q], g.sx, x[q], &special), g.hsx, y[q], &special);
                    }
#pragma unroll
                    for (int q = 0; q < NQ; q++)
                        u[q] = special ? sub_half_scaled(sub_scaled(u[q], g.sx, x[q]), g.hsx, y[q]) : v[q];
                }
            }
        }
        // the next sweep's windows reach H cells into this chunk; after the last sweep, all of it
        const bool done = (sweep + 1) * A.S >= A.steps;
        if (own && writes && (done || i < a + H || i >= b - H)) {
#pragma unroll
            for (int q = 0; q < NQ; q++) Uout[(long)(q0 + q) * n + i] = u[q];
        }
        if (!done) {
            __syncthreads();
            // (the barrier orders the block's stores before the release)
            if (threadIdx.x == 0 && c != A.stall)
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(A.prog + c * kPlainProgStride),
                             "r"((unsigned)(sweep + 1)) : "memory");
        }
    }
    if (bad) atomicOr(A.flag, SHLL_FLAG_NONPOSITIVE);
}

// ---------------- host ----------------
struct ResPlan {
    int chunks, threads, S, lanes;
    bool resident;
};

// Chunks, window and steps per sweep.  One chunk per SM where the windows fit; then the window of
// least estimated time per step: the step's chain (`chain` clocks) plus a share per warp (`share`), or,
// where it is more, the block's instruction time (`work` clocks per warp: FP64 about 42 + 10 instructions
// of 19 clocks for order 1, 70 + 12 for order 2), plus the exchange (about 4500 clocks) over the S steps
// it serves.  A narrower window means less redundant work per step, a wider one fewer exchanges.
// Measured, us a step with 32 / 64 / 96 / 128 / 256 / 512 threads at 1024 cells: FP64 first order 1.70 /
// 1.64 / 1.62 / 1.66 / 2.10 / 3.11, float 0.53 / 0.47 / 0.45 / 0.44 / 0.45 / 0.51 (0.40 with the present cell1).
template <typename REAL, int ORDER>
static ResPlan res_plan(int n, long steps, int sms) {
    const bool wide = sizeof(REAL) == 8;
    const double chain = wide ? (ORDER == 1 ? 3000 : 5200) : (ORDER == 1 ? 800 : 1450);
    const double share = wide ? (ORDER == 1 ? 300 : 450) : (ORDER == 1 ? 30 : 45);
    const double work = wide ? (ORDER == 1 ? 1000 : 1560) : (ORDER == 1 ? 70 : 110);
    ResPlan best = {0, 0, 0, 1, false};
    double best_t = 1e30;
    const int k = std::min(sms, n);
    const int owned = (n + k - 1) / k;
    for (int T = 64; T <= kResThreads; T += 32) {
        const int S = (int)std::min<long>((T - owned) / (2 * ORDER), steps);
        if (S < 1) continue;
        const double warps = (owned + ORDER * (S + 1)) / 32.0 + 0.5;
        const double t = std::max(chain + (warps + std::max(0, T / 32 - 4) * 0.5) * share, warps * work) +
                         (wide ? 3000.0 : 4500.0) / S;
        if (t < best_t) { best_t = t; best = {k, T, S, 1, true}; }
    }
    // FP64 with four lanes per cell: a shorter chain, more FP64 instructions in all (1024 cells: first order
    // 1.62 -> 1.26 us a step, second 2.80 -> 1.82; from 8192 cells on one lane per cell is faster, first order
    // 1.67 against 2.08)
    if (wide) {
        for (int T = 128; T <= 256; T += 64) {
            const int S = (int)std::min<long>((T / 4 - owned) / (2 * ORDER), steps);
            if (S < 1) continue;
            const double warps = 4 * (owned + ORDER * (S + 1)) / 32.0;
            const double t = (ORDER == 1 ? 2200 : 3400) + std::max(0.0, warps - 3.0) * (ORDER == 1 ? 300 : 450) +
                             std::max(0, T / 32 - 4) * 60.0 + 3000.0 / S;
            if (t < best_t) { best_t = t; best = {k, T, S, 4, true}; }
        }
    }
    // more cells than one window per SM holds (or windows with hardly any margin): several blocks per
    // SM, one launch per sweep of 8 steps
    if (best.chunks == 0 || (best.S < 4 && best.lanes == 1)) {
        const int T = 256, S = (int)std::min<long>(8, steps), per = T - 2 * ORDER * S;
        best = {(n + per - 1) / per, T, S, 1, false};
    }
    return best;
}

template <typename REAL, int ORDER>
static cudaError_t run1_t(const PlainArgs& a, long steps, unsigned* prog, int stall, int* swaps) {
    int dev = 0, sms = 1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    ResPlan p = res_plan<REAL, ORDER>(a.nx, steps, std::min(sms, kPlainProgChunks));
    auto* kern = k_resident1<REAL, ORDER, 1>;
    if constexpr (sizeof(REAL) == 8) {
        if (p.lanes == 4) kern = k_resident1<REAL, ORDER, 4>;
    }
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)res_smem<REAL, ORDER>(kResThreads));
    if (e != cudaSuccess) return e;
    const size_t smem = res_smem<REAL, ORDER>(p.threads / p.lanes);
    const Gas<REAL> g = make_gas<REAL>(a);
    ResArgs<REAL> A;
    A.U[0] = static_cast<REAL*>(const_cast<void*>(a.Uin));
    A.U[1] = static_cast<REAL*>(a.Uout);
    A.n = a.nx;
    A.S = p.S;
    A.steps = steps;
    A.prog = prog;
    A.flag = a.flag;
    A.stall = stall;
    const long sweeps = (steps + p.S - 1) / p.S;
    if (p.resident && sweeps > 1) {   // every block must be resident at once
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, p.threads, smem);
        if (e != cudaSuccess) return e;
        p.resident = prog && (long)per_sm * sms >= p.chunks;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.chunks);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = a.stream;
    if (sweeps == 1 || p.resident) {
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = sweeps > 1 ? 1 : 0;
        if (sweeps > 1)
            e = cudaMemsetAsync(prog, 0, sizeof(unsigned) * kPlainProgStride * p.chunks, a.stream);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, A, g);
        shll_count_launches(1);
    } else {
        A.prog = nullptr;
        for (long q = 0; q < sweeps && e == cudaSuccess; q++) {
            A.steps = std::min<long>(p.S, steps - q * p.S);
            e = cudaLaunchKernelEx(&cfg, kern, A, g);
            shll_count_launches(1);
            std::swap(A.U[0], A.U[1]);
        }
    }
    *swaps = (int)(sweeps & 1);
    return e;
}

// `steps` time steps of a 1D problem from Uin; *swaps = 1 when the result lies in Uout
template <typename REAL>
static cudaError_t run_t(const PlainArgs& a, long steps, unsigned* prog, int stall, int* swaps) {
    return a.order == 1 ? run1_t<REAL, 1>(a, steps, prog, stall, swaps) : run1_t<REAL, 2>(a, steps, prog, stall, swaps);
}

}  // namespace SHLL_PLAIN_NS
