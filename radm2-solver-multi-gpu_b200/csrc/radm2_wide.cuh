// The wide tensor-memory solver: FP64 ROS-3, one cell per thread, one 128-thread CTA per SM,
// cells from a work queue.  The same step loop as k_rosenbrock (radm2_solver.cuh): time-loop
// mask and step clamp (mgpu.cu:1595-1614), Jacobian and matrix (mgpu.cu:1672-2652, 3128-3166),
// pivot-free LU (mgpu.cu:2726-2780), three ROS-3 stages (mgpu.cu:3595-3625, restored), error
// norm and step-size control (mgpu.cu:3168-3262), with the operations on each value in the
// same order.  ARITH 0: reciprocal pivots, the compiler's multiply-add contraction; 1: the
// reference's divisions, built without contraction.
//
// What bounds it and why it is built this way (B200, 262,144 mixed cells, one 600 s step):
//   Instruction fetch.  A step attempt is straight-line code (200 KB), so an SM streams all of
//   it once per attempt.  Measured on straight-line code beyond 128 KB: 6.1 cycles per
//   instruction for one warp, the same for 4 or 8 warps that run the same lines together, 12.5
//   for 4 warps on lines of their own.  So fewer instructions are faster whatever they do: the
//   RHS and the solve exist once and run in a loop over the stages, and the error norm is a
//   small loop.  Keeping the warps together costs more than it gives: a block-wide vote per
//   attempt takes 86 ms instead of 83, barriers inside the phases 90-110 ms.
//   Memory latency.  One warp per scheduler hides nothing, so the generated phases issue
//   their global loads about 100 operations ahead and each tensor-memory group while the
//   previous one is used.
//   L2 capacity.  Reads from the scratch run at 12 TB/s while all SMs' scratch stays under
//   75 MB, 8 TB/s at 100 MB, 4 TB/s at 160 MB (measured).  Per thread: shared memory holds the
//   state, the 88 distinct rate constants and 79 LU slots, tensor memory 256 LU slots, global
//   scratch 501 words (76 MB over 148 SMs).
#pragma once

#include "gen/radm2_wide_map.h"
#include "gen/radm2_wide_tmem.h"
#include "radm2_div.cuh"
#include "radm2_internal.h"

namespace radm2 {

constexpr int WIDE_BS = 128;
#if RADM2_WIDE_DIV
constexpr int WIDE_GLOBAL_WORDS = RADM2_WIDE_GLOBAL_WORDS_DIV;
#else
constexpr int WIDE_GLOBAL_WORDS = RADM2_WIDE_GLOBAL_WORDS;
#endif
constexpr int WIDE_SMEM_BYTES = RADM2_WIDE_SMEM_WORDS * WIDE_BS * 8;
static __constant__ unsigned char c_wide_rc_rep[RADM2_WIDE_RC_WORDS] = RADM2_WIDE_RC_REP_INIT;

#if RADM2_WIDE_DIV
// limit: -1 once a pivot of this attempt has no reciprocal, so that all its divisions are plain
#define DIVR(a, u, r) div_pivot(a, u, r, limit)
#define RCPR(u) [&](double r_) { limit = r_ != r_ ? -1.0f : limit; return r_; }(rcp_pivot(u))
#endif

// Global scratch, word w of the thread (1 KB apart, so every access of a warp is 256 bytes
// together).  Volatile statements keep the order in which the generated code issues them;
// the I forms take an index that only unrolling makes constant.
#define GLD(v, w) asm volatile("ld.global.f64 %0, [%1+%2];" : "=d"(v) : "l"(gp), "n"((w) * WIDE_BS * 8))
#define GST(w, v) asm volatile("st.global.f64 [%0+%1], %2;" ::"l"(gp), "n"((w) * WIDE_BS * 8), "d"(v))
#define GLDI(v, p, w) asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"((p) + (w) * WIDE_BS))
#define GSTI(w, v) asm volatile("st.global.f64 [%0], %1;" ::"l"(gp + (w) * WIDE_BS), "d"(v))
// Shared memory, word k of the thread: state (or stage input), rate constants, LU slots.
#define SL(k) sm[(k) * WIDE_BS]
#define V(i) sm[(i) * WIDE_BS]
#define RC(k) sm[(NVAR + (k)) * WIDE_BS]
#define FIX(k) ((k) == 0 ? fix0 : fix1)
#define X(i) x[i]
#define TM_BASE tb

template <int ARITH>
__global__ void __launch_bounds__(WIDE_BS, 1) k_rosenbrock_wide(const SolveArgs a)
{
    extern __shared__ double smem[];
    __shared__ uint32_t tmem_base;
    if (threadIdx.x < 32) {  // all 512 columns; the permit is given up, as nothing more is allocated
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t talloc = tmem_base;
    const uint32_t tb = talloc + ((threadIdx.x & 96u) << 16);  // warp w: lanes 32 w .. 32 w + 31
    double *const sm = smem + threadIdx.x;
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(sm);
    double *const gp = a.scratch + (size_t)blockIdx.x * (WIDE_GLOBAL_WORDS * WIDE_BS) + threadIdx.x;
    const SolveParams &P = a.p;
    const int ld = a.ld;
    const int dir = P.direction;

    // ---- lane state; a lane starts as one whose (absent) cell is done
    int cidx = -1;
    bool have = a.warps == 0 || (int)threadIdx.x < 32 * a.warps;
    bool outer = true, done = true;
    double T = 0.0, H = 1.0, fix0 = 0.0, fix1 = 0.0, hfirst = 0.0;
    int rlast = 0, rmore = 0, nacc = 0, nrej = 0, nstp = 0, status = 1;

    // The lane's next cell: the warp's lanes that need one take consecutive ones.  Its arrays
    // go to shared memory by asynchronous copies (no registers, all in flight together).
    auto take_cell = [&]() {
        const unsigned m = __activemask();
        const int lane = threadIdx.x & 31;
        const int leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(a.queue, __popc(m));
        base = __shfl_sync(m, base, leader);
        const int cell = base + __popc(m & ((1u << lane) - 1));
        have = cell < a.ncell;
        if (!have) return;
        cidx = a.order ? a.order[cell] : cell;
        const double *v = a.var + cidx;
#pragma unroll 8
        for (int i = 0; i < NVAR; i++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa + i * (WIDE_BS * 8)),
                         "l"(v + (size_t)i * ld)
                         : "memory");
        const double *rc = a.rconst + cidx;
#pragma unroll 8
        for (int k = 0; k < RADM2_WIDE_RC_WORDS; k++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa + (NVAR + k) * (WIDE_BS * 8)),
                         "l"(rc + (size_t)(a.rc_words ? k : c_wide_rc_rep[k]) * ld)
                         : "memory");
        fix0 = a.fix[cidx];
        fix1 = a.fix[(size_t)ld + cidx];
        T = P.Tstart;
        double hs = P.Hstart;
        if (a.h0) {
            const double h = a.h0[cidx];
            if (h > 0.0 && h <= P.Hmax) hs = h;  // non-finite or out of range: default
        }
        H = mind(hs, P.Hmax);  // mgpu.cu:3475-3477
        if (absd(H) <= 10.0 * P.Roundoff) H = DELTA_MIN;
        rlast = rmore = nacc = nrej = nstp = 0;
        status = 1;
        hfirst = 0.0;
        outer = true;
        done = false;
        asm volatile("cp.async.wait_all;" ::: "memory");
    };
    auto store_cell = [&]() {
        double *v = a.var + cidx;
#pragma unroll
        for (int i = 0; i < NVAR; i++) v[(size_t)i * ld] = SL(i);
        a.status[cidx] = status;
        a.nacc[cidx] = nacc;
        a.nrej[cidx] = nrej;
        a.hfirst[cidx] = hfirst;
        a.hexit[cidx] = H;
        a.texit[cidx] = T;
    };

    for (int k = 0; k < NVAR + RADM2_WIDE_RC_WORDS; k++) SL(k) = 0.0;  // for a lane that never gets a cell

    for (;;) {
        // Bring every lane that still has work to the start of a step attempt.
        while (have && (outer || done)) {
            if (done) {
                if (cidx >= 0) store_cell();
                take_cell();
                continue;
            }
            // Time-loop mask (mgpu.cu:1608-1613).
            const bool more = (dir > 0 && (T - P.Tend) + P.Roundoff <= 0.0) ||
                              (dir < 0 && (P.Tend - T) + P.Roundoff <= 0.0);
            if (!more) {
                done = true;
                continue;
            }
            H = mind(H, absd(P.Tend - T));
            outer = false;
        }
        if (!__any_sync(0xffffffffu, have)) break;

        // ---------------------------------------------------------------- one attempt
        // Every lane runs it (tensor-memory accesses are warp-collective); a lane without an
        // attempt (act false) runs it on its own words and keeps its state.
        bool act = have;
        if (act && nstp >= P.max_steps) {
            status = -6;
            done = true;
            act = false;
        }
        if (act && ((T + 0.1 * H == T) || (H <= P.Roundoff))) {
            status = -7;
            done = true;
            act = false;
        }
        const double Ha = act ? H : 1.0;
        const double ghinv = 1.0 / (dir * Ha * RADM2_ROS_GAMMA0);
        __syncwarp();
        {
#include "gen/radm2_wide_jac.inc"
        }
        // LU; a zero pivot is looked for before its row is eliminated (mgpu.cu:2753-2757).  The
        // pivots of rows without eliminations lie side by side and are inverted in a loop.
        bool sing = false;
#if RADM2_WIDE_DIV
        float limit = PIVOT_MAX;
#endif
#define LU_PIVOT_CHECK(v) sing = sing | ((v) == 0.0)
#pragma unroll 4
        for (int k = 0; k < RADM2_WIDE_SPIVOTS; k++) {
            const double v = SL(RADM2_WIDE_SPIVOT + k);
            LU_PIVOT_CHECK(v);
#if RADM2_WIDE_DIV
            GSTI(RADM2_WIDE_GRCP + k, RCPR(v));
#else
            SL(RADM2_WIDE_SPIVOT + k) = 1.0 / v;
#endif
        }
        __syncwarp();
        {
#if RADM2_WIDE_DIV
#include "gen/radm2_wide_lu.inc"
#else
#include "gen/radm2_wide_lu_rcp.inc"
#endif
        }
#undef LU_PIVOT_CHECK
        if (act && sing) {
            status = -8;
            done = true;
            act = false;
        }

        // Stages.  x holds a stage's right-hand side, then its K.
        //   0: F(Y)                       -> K1
        //   1: F(Y + A21 K1) + C21/h K1   -> K2   (the state makes room for the stage input)
        //   2: F (of stage 1) + C31/h K1 + C32/h K2 -> K3, its first two terms kept in V
        const double hc21 = RADM2_ROS_C0 / (dir * Ha);
        const double hc31 = RADM2_ROS_C1 / (dir * Ha);
        const double hc32 = RADM2_ROS_C2 / (dir * Ha);
        double x[NVAR];
#pragma unroll 1
        for (int stage = 0; stage < 3; stage++) {
            __syncwarp();
            if (stage == 1) {
#pragma unroll
                for (int i = 0; i < NVAR; i++) {
                    const double y = V(i);
                    GSTI(RADM2_WIDE_GK1 + i, x[i]);
                    GSTI(RADM2_WIDE_GY + i, y);
                    V(i) = y + RADM2_ROS_A0 * x[i];
                }
            }
            if (stage < 2) {
#include "gen/radm2_wide_fun.inc"
#pragma unroll
                for (int i = 0; i < NVAR; i++) asm volatile("" : "+d"(x[i]));  // F is rounded before it is used
            }
            if (stage == 1) {
                constexpr int A = 30;  // loads in flight
                double k1[NVAR];
#pragma unroll
                for (int i = 0; i < NVAR + A; i++) {
                    if (i < NVAR) GLDI(k1[i], gp, RADM2_WIDE_GK1 + i);
                    if (i >= A) {
                        const double f = x[i - A];
                        x[i - A] = f + k1[i - A] * hc21;
                        V(i - A) = f + k1[i - A] * hc31;
                    }
                }
            }
            if (stage == 2) {
#pragma unroll
                for (int i = 0; i < NVAR; i++) {
                    GSTI(RADM2_WIDE_GK2 + i, x[i]);
                    x[i] = V(i) + x[i] * hc32;
                }
            }
            __syncwarp();
#if RADM2_WIDE_DIV
#include "gen/radm2_wide_solve.inc"
#else
#include "gen/radm2_wide_solve_rcp.inc"
#endif
        }

        // New state (into V) and error norm (mgpu.cu:3223-3238), U species at a time, the next
        // ones' K1, K2 and state being loaded meanwhile.  The sum is in species order.  A
        // division takes 141 cycles and they follow one another, so four species share one
        // (262,144 cells x 2 steps 116.5 ms, 119.2 with one each).
#pragma unroll
        for (int i = 0; i < NVAR; i++) V(i) = x[i];  // K3
        double err = 0.0;
        {
            constexpr int U = 4, END = (NVAR + U - 1) / U * U;
            static_assert(END - NVAR < U && RADM2_WIDE_GY + END <= WIDE_GLOBAL_WORDS && END <= NTOL,
                          "the last step reads past the species");
            double k0[U], k1[U], y[U];
            const double *g = gp;
            auto load = [&]() {
#pragma unroll
                for (int j = 0; j < U; j++) {
                    GLDI(k0[j], g, RADM2_WIDE_GK1 + j);
                    GLDI(k1[j], g, RADM2_WIDE_GK2 + j);
                    GLDI(y[j], g, RADM2_WIDE_GY + j);
                }
                g += U * WIDE_BS;
            };
            load();
#pragma unroll 1
            for (int i = 0; i < END; i += U) {
                double num[U], den[U], q[U];
#pragma unroll
                for (int j = 0; j < U; j++) {
                    const bool in = j < U - (END - NVAR) || i + j < NVAR;  // the last step is not full
                    const double k2 = V(i + j);
                    const double ynew = P.M[0] * k0[j] + P.M[1] * k1[j] + P.M[2] * k2 + y[j];
                    const double yerr = P.E[0] * k0[j] + P.E[1] * k1[j] + P.E[2] * k2;
                    const double ymax = maxd(fabs(y[j]), fabs(ynew));
                    const double scale = P.AbsTol[i + j] + P.RelTol[i + j] * ymax;
                    num[j] = in ? yerr * yerr : 0.0;
                    den[j] = in ? scale * scale : 1.0;
                    if (in) V(i + j) = ynew;
                }
                if (i + U < END) load();
                div_four(num, den, q);
#pragma unroll
                for (int j = 0; j < U; j++) err += q[j];
            }
        }

        // Step control (mgpu.cu:3240-3260).
        bool take = false;
        if (act) {
            nstp++;
            err = sqrt(err / (double)NVAR);
            const double fac = mind(P.FacMax, maxd(P.FacMin, P.FacSafe / pow(err, 1.0 / RADM2_ROS_ELO)));
            double hnew = H * fac;
            if (err != err) hnew = H * P.FacRej;  // non-finite norm: shrink hard and retry
            take = (err <= 1.0) || (H <= P.Hmin);
            if (take) {
                T += dir * H;
                if (rlast) hnew = mind(hnew, H);
                rlast = 0;
                rmore = 0;
                if (nacc == 0) hfirst = H;
                nacc++;
                H = hnew;
                outer = true;
            } else {
                if (rmore) hnew = H * P.FacRej;
                rmore = rlast;
                rlast = 1;
                nrej++;
                H = hnew;
            }
        }
        if (!take) {  // the state back in its place
#pragma unroll
            for (int i = 0; i < NVAR; i++)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa + i * (WIDE_BS * 8)),
                             "l"(gp + (RADM2_WIDE_GY + i) * WIDE_BS)
                             : "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
    }
    // every warp is done with its tensor memory: warp 0 frees it
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(talloc), "r"(512u) : "memory");
}

#undef TM_BASE
#undef X
#undef FIX
#undef RC
#undef V
#undef SL
#undef GSTI
#undef GLDI
#undef GST
#undef GLD

template <int ARITH>
cudaError_t launch_wide(const SolveArgs &a, int grid, cudaStream_t st)
{
    auto k = k_rosenbrock_wide<ARITH>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, WIDE_SMEM_BYTES);
    if (e != cudaSuccess) return e;
    (void)cudaGetLastError();  // a stale error from another library is not this launch's
    k<<<grid, WIDE_BS, WIDE_SMEM_BYTES, st>>>(a);
    return cudaGetLastError();
}

template <int ARITH>
cudaError_t info_wide(SolverInfo *out)
{
    auto k = k_rosenbrock_wide<ARITH>;
    cudaFuncAttributes at{};
    cudaError_t e = cudaFuncGetAttributes(&at, k);
    if (e != cudaSuccess) return e;
    out->regs = at.numRegs;
    out->local_bytes = (int)at.localSizeBytes;
    out->blocks_per_sm = 1;  // all of an SM's tensor memory
    out->global_words = WIDE_GLOBAL_WORDS;
    out->smem_bytes = WIDE_SMEM_BYTES;
    return cudaSuccess;
}

}  // namespace radm2
