/* The OdeVec BDF integrator as one persistent CUDA kernel (sm_100a).
 *
 * One thread integrates one cell.  A warp is either 32 independent cells
 * (G = 1: per-cell time, step, order and Jacobian decisions) or one lockstep
 * group of 32 cells that share them through max-norms over the warp
 * (G = 32: the reference's semantics with nvector = 32, with warp
 * reductions).  The grid is persistent: idle lanes take the next cells
 * from a global counter (warp-aggregated atomicAdd), so a warp keeps its
 * lanes busy while cells of very different stiffness finish at different
 * times.
 *
 * The reference's nested loops (src/odevec.F90: step loop :207, predictor
 * retry loop :259, corrector loop :321) are flattened into a per-lane state
 * machine.  Each trip of the main loop performs for every lane at most one
 * predictor, one right-hand-side evaluation and one Newton update, so lanes
 * in different phases still run the right-hand side and the solve together.
 * The two expensive and rarely needed blocks -- Jacobian + LU factorisation
 * and step-size/order selection -- exist once in the code; a lane that needs
 * one waits, and all waiting lanes run it together: on staging 1 once enough
 * lanes of its warp need it (jac_batch / ss_batch), no lane can progress
 * otherwise, or it has waited max_wait trips; on the other stagings on fixed
 * trips (StageCfg::PERIOD), the same trips in every warp of the block, so a
 * trip runs at most one of the two and all warps run the same code.  Waiting
 * changes only the interleaving
 * across lanes, never a cell's own sequence of operations: the arithmetic
 * per cell is that of src/odevec.F90 operation by operation, and with
 * --fmad=false it is bit-identical to the CPU oracle.
 *
 * Species whose right-hand side is identically zero and on which nothing
 * depends (the network header's frozen(); PRIMORDIAL's CR, g, Tgas, dummy)
 * are not part of the solver state: their corrections are exact zeros in
 * the reference, so leaving them out changes no result.  Norms still divide
 * by the full neq.
 *
 * Per-cell state: en, en_old, error weights, the state and the packed LU in
 * thread-local arrays with compile-time indices (the LU in shared memory for
 * stagings 2, 5, 11 and 22, the launcher's own); the Nordsieck history
 * y_NS(0:5), which loops over the runtime order index, in a thread-local array
 * or, for stagings 2, 5, 9-12, 17, 21 and 22, in shared memory laid out
 * [entry][lane]; up to four species it stays in registers elsewhere.  The staging (StageCfg) also
 * fixes the block size, the blocks per SM, whether the block's warps run in
 * soft lockstep and how often idle lanes take new cells.
 *
 * Every loop is bounded: at most max_attempts predictor attempts per cell
 * (status OV_ERR_MAX_STEPS), at most 4 Newton iterations per attempt and 10
 * consecutive Newton failures (OV_ERR_CONV_FAILURES), so a stiff or broken
 * cell ends with a status code instead of holding the GPU. */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/odevec_b200.h"
#include "ov_common.h"
#include "ov_host.h"
#include "ov_launch.h"
#include "rates_primordial.h"

#ifndef OV_MODE_NS
#error "OV_MODE_NS (the arithmetic-mode namespace) must be defined"
#endif

namespace ov {
namespace OV_MODE_NS {

constexpr int MAXQ = 5; /* maxorder, pre_odevec.py:83 */
constexpr unsigned FULL = 0xffffffffu;

enum Phase : int {
    PH_IDLE = 0,      /* no cell */
    PH_START = 1,     /* cell loaded: initial right-hand side pending */
    PH_PRED = 2,      /* next: predictor attempt */
    PH_JACWAIT = 3,   /* predicted; waits for the Jacobian + LU block */
    PH_NEWTON = 4,    /* next: right-hand side + Newton update */
    PH_RESTART = 5,   /* next: right-hand side at the predicted state (3 error-test failures) */
    PH_SSWAIT = 6,    /* waits for the step-size/order selection block */
    PH_DONE = 7,      /* finished (status says how) */
    PH_EXHAUSTED = 8  /* no cells left */
};

/* why a lane waits for the step-size selection */
enum SsMode : int { SS_REJECT = 1, SS_RESTART = 2, SS_ACCEPT = 3 };

/* Nordsieck l-vectors l(q, 0:q), q = 1..6 (src/odevec.F90:127-134) */
static __constant__ double c_lcoef[7][7] = {
    {0, 0, 0, 0, 0, 0, 0},
    {1.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0},
    {2.0 / 3.0, 1.0, 1.0 / 3.0, 0.0, 0.0, 0.0, 0.0},
    {6.0 / 11.0, 1.0, 6.0 / 11.0, 1.0 / 11.0, 0.0, 0.0, 0.0},
    {12.0 / 25.0, 1.0, 7.0 / 10.0, 1.0 / 5.0, 1.0 / 50.0, 0.0, 0.0},
    {60.0 / 137.0, 1.0, 225.0 / 274.0, 85.0 / 274.0, 15.0 / 274.0, 1.0 / 274.0, 0.0},
    {20.0 / 49.0, 1.0, 58.0 / 63.0, 5.0 / 12.0, 25.0 / 252.0, 1.0 / 84.0, 1.0 / 1764.0}};

__device__ __forceinline__ double lcoef(int q, int k) { return c_lcoef[q][k]; }

/* 1/k for k = 1..7, correctly rounded at compile time: the same bits as the
   division 1.0 / k the reference evaluates (1/order, 1/(order+1), ...) */
static __constant__ double c_inv[8] = {0.0, 1.0, 1.0 / 2.0, 1.0 / 3.0, 1.0 / 4.0, 1.0 / 5.0, 1.0 / 6.0, 1.0 / 7.0};

/* tau (src/odevec.F90:1034-1054), evaluated at compile time with the same
   IEEE operations: q! by repeated multiplication, then one division */
constexpr double kL[7] = {0.0, 1.0, 1.0 / 3.0, 1.0 / 11.0, 1.0 / 50.0, 1.0 / 274.0, 1.0 / 1764.0};
constexpr double tau_c(int order, int order2)
{
    double faculty = 1.0;
    for (int i = 1; i <= order; ++i)
        faculty = faculty * i;
    if (order - 1 == order2)
        return (order2 + 1.0) / faculty;
    return (order2 + 1.0) / (faculty * kL[order]);
}
/* per order q = 1..5: tau(q,q-1), tau(q,q), tau(q,q+1) and the
   convergence-test divisor tau(q,q) / (2 (q+2)) (src/odevec.F90:640-641) */
static __constant__ double c_tau[6][4] = {
    {0, 0, 0, 0},
#define OV_TAU_ROW(q) {tau_c(q, q - 1), tau_c(q, q), tau_c(q, q + 1), tau_c(q, q) / (2.0 * (q + 2.0))}
    OV_TAU_ROW(1), OV_TAU_ROW(2), OV_TAU_ROW(3), OV_TAU_ROW(4), OV_TAU_ROW(5)
#undef OV_TAU_ROW
};
__device__ __forceinline__ double tau(int order, int order2) { return c_tau[order][order2 - order + 1]; }
__device__ __forceinline__ double conv_divisor(int order) { return c_tau[order][3]; }

/* per order q: the smallest double x with sqrt(x) / tau(q,q) > 1 in double
   arithmetic, i.e. whose rounded root exceeds tau(q,q).  The local error
   test norm / tau > 1 (src/odevec.F90:402-404) then needs neither the root
   nor the division: both are monotone, so comparing the norm's square with
   this bound decides the same way for every input */
static __constant__ double c_lte[6] = {0.0, 0x1.0000000000002p+2, 0x1.4400000000002p+4, 0x1.ae38e38e38e3cp+5,
                                       0x1.b2071c71c71cbp+6, 0x1.776147ae147b0p+7};

/* NaN and masked-out values never win a max (as the oracle's comparison loop) */
__device__ __forceinline__ double max_operand(double v) { return v > -HUGE_VAL ? v : -HUGE_VAL; }

/* Correctly rounded reciprocal of x in [2^-1000, 2^1000) whose significand is
   not all ones: Newton's iteration from the hardware estimate, the last step
   with the residual formed exactly by a fused multiply-add, which rounds
   correctly for these x (P. Markstein, "Computation of elementary functions
   on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990,
   theorem 8.3).  No branch: independent reciprocals interleave. */
__device__ __forceinline__ double rcp_normal(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = __fma_rn(__fma_rn(-x, r, 1.0), r, r);
    r = __fma_rn(__fma_rn(-x, r, 1.0), r, r);
    r = __fma_rn(__fma_rn(-x, r, 1.0), r, r);
    return r;
}
/* nonzero for the x that rcp_normal does not cover (or might not) */
__device__ __forceinline__ unsigned rcp_odd(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    return (hi - (23u << 20) >= (2000u << 20)) | (lo == 0xffffffffu);
}

template <int G>
__device__ __forceinline__ double group_max(double v)
{
    v = max_operand(v);
    if (G == 32) {
        /* v is -infinity or non-negative, so its words order as integers:
           the largest upper word, then the largest lower word beside it.  Two
           integer reductions instead of ten shuffles and five comparisons */
        const int hi = __double2hiint(v);
        const int top = __reduce_max_sync(FULL, hi);
        const unsigned low = __reduce_max_sync(FULL, hi == top ? (unsigned)__double2loint(v) : 0u);
        v = __hiloint2double(top, (int)low);
    }
    return v;
}

template <int G>
__device__ __forceinline__ bool group_any(bool b)
{
    if (G == 32)
        return __any_sync(FULL, b);
    return b;
}

/* The choice of CalcStepSizeOrder (src/odevec.F90:547-618) from the squared
   norms of the three candidates (x_down read only with has_down, x_up only
   with has_up): returns the step-size factor; loc = 1, 2, 3 for order - 1,
   the same order and order + 1, big when the factor reaches 1.1, so that the
   order changes.  The literals 1.3, 1.2, 1.4 and 1.1 are single precision in
   the reference.

   Of the three candidate factors only one is used: the largest if it reaches
   1.1, else the one of the same order.  Which one that is follows from
   single-precision estimates (relative error below 1e-4) unless two
   candidates, or the largest and 1.1, lie within 1e-3 of each other; then all
   are evaluated.  So a lane evaluates one root, quotient and power instead of
   three, each kept value the same IEEE expression as in the reference.  Bound
   by the chain of dependent FP64 operations of a power (1,048,576 PRIMORDIAL
   cells with FP32 factors: 109.3 -> 107.4 ms; a lockstep group evaluated three
   powers one after another). */
__device__ __forceinline__ double step_choice(int order, bool has_down, bool has_up, double x_down, double x_same,
                                              double x_up, int& loc_out, bool& big_out)
{
    /* candidate loc = 1, 2, 3: 1 / (c * (norm / tau)^(1/k) + 1e-6) */
    auto factor = [&](int loc) {
        const double x = loc == 1 ? x_down : (loc == 2 ? x_same : x_up);
        const double cc = loc == 1 ? (double)1.3f : (loc == 2 ? (double)1.2f : (double)1.4f);
        const double n = (x < 0.0 ? x : sqrt(x)) / c_tau[order][loc - 1];
        return 1.0 / (cc * ov_pow_sel(n, c_inv[order + loc - 1]) + 1e-6);
    };
    auto estimate = [&](double x, float cc, int loc) {
        const int hi = __double2hiint(x);
        const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3));
        const float l = (float)((hi >> 20) - 1023) + __log2f(m);
        return cc * exp2f((0.5f * l - __log2f((float)c_tau[order][loc - 1])) * (float)c_inv[order + loc - 1])
               + 1e-6f;
    };
    const float e_same = estimate(x_same, 1.2f, 2);
    const float e_down = has_down ? estimate(x_down, 1.3f, 1) : HUGE_VALF;
    const float e_up = has_up ? estimate(x_up, 1.4f, 3) : HUGE_VALF;
    const float best = fminf(e_same, fminf(e_down, e_up));
    const float near_best = best * 1.001f;
    const bool one_best = (e_same <= near_best) + (e_down <= near_best) + (e_up <= near_best) == 1;
    const bool below = best * 1.1f > 1.001f; /* the largest factor is below 1.1 */
    const bool above = best * 1.1f < 0.999f;
    /* infinities and NaN (a negative squared norm) take the full comparison */
    const bool finite = x_same >= 0.0 && x_same < HUGE_VAL && (!has_down || (x_down >= 0.0 && x_down < HUGE_VAL))
                        && (!has_up || (x_up >= 0.0 && x_up < HUGE_VAL));
    const bool clear = finite && (below || (above && one_best));
    int loc = 2;
    if (clear && above)
        loc = e_down <= near_best ? 1 : (e_up <= near_best ? 3 : 2);
    double s = factor(loc);
    bool big = above;
    if (!clear) {
        const double same = s;
        const double down = has_down ? factor(1) : 0.0;
        const double up = has_up ? factor(3) : 0.0;
        loc = 1;
        double mx = down;
        if (same > mx) { mx = same; loc = 2; }
        if (up > mx) { mx = up; loc = 3; }
        big = mx >= (double)1.1f;
        s = big ? mx : same;
    }
    loc_out = loc;
    big_out = big;
    return s;
}

/* Shared-memory staging: per-lane arrays laid out [entry][lane] with a
   stride of the block size, so a warp's 32 lanes touch 32 consecutive
   words (no bank conflicts). */
template <class T, int BS>
struct LaneCol {
    T* base; /* &array[0][threadIdx.x] */
    __device__ __forceinline__ T& operator[](int i) const { return base[i * BS]; }
};

template <int ND, int BS>
struct LaneHist {
    double* base;
    __device__ __forceinline__ LaneCol<double, BS> operator[](int k) const
    {
        return LaneCol<double, BS>{base + k * ND * BS};
    }
};

/* Kernel configurations ("stagings"): where the per-cell arrays live and the
   launch shape.  BS threads per block, MINB blocks per SM for the register
   budget; SHM places the Nordsieck history and the LU in shared memory. */
template <int STAGE>
struct StageCfg;
/* SHM: 0 = history and LU in thread-local arrays, 1 = both in shared memory,
   2 = the history in shared memory and the LU thread-local.  REFILL: idle
   lanes take new cells on every REFILL-th trip of the cell loop only (the
   first trip included), so a warp sets up several cells at once instead of
   one every few trips, and the lockstep stagings set up cells in all their
   warps in the same trip.  PERIOD > 1: the Jacobian + LU block runs on the
   trips t with t % PERIOD == 1 and the step-size block on those with
   t % PERIOD == 0 (or at once when no lane of the warp can progress
   otherwise), the same trips in every warp; jac_batch / ss_batch / max_wait
   apply with PERIOD = 1 only. */
/* staging 1 keeps the straight port's refill on every trip */
template <> struct StageCfg<1> { static constexpr int SHM = 0; static constexpr bool SOFT = false; static constexpr int BS = 128, MINB = 2, REFILL = 1, PERIOD = 1; };
template <> struct StageCfg<2> { static constexpr int SHM = 1; static constexpr bool SOFT = false; static constexpr int BS = 128, MINB = 1, REFILL = 16, PERIOD = 4; };
template <> struct StageCfg<3> { static constexpr int SHM = 0; static constexpr bool SOFT = false; static constexpr int BS = 128, MINB = 3, REFILL = 16, PERIOD = 4; };
template <> struct StageCfg<4> { static constexpr int SHM = 0; static constexpr bool SOFT = false; static constexpr int BS = 128, MINB = 4, REFILL = 16, PERIOD = 4; };
template <> struct StageCfg<5> { static constexpr int SHM = 1; static constexpr bool SOFT = false; static constexpr int BS = 192, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 3, the same register budget, in one block of 384 threads per SM */
template <> struct StageCfg<6> { static constexpr int SHM = 0; static constexpr bool SOFT = false; static constexpr int BS = 384, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 6, with the block's warps held in soft lockstep (SoftSync) */
template <> struct StageCfg<8> { static constexpr int SHM = 0; static constexpr bool SOFT = true;  static constexpr int BS = 384, MINB = 1, REFILL = 16, PERIOD = 4; };
/* soft lockstep, one block of 256 threads per SM, the history in shared
   memory (the rest of L1 for the other per-cell arrays) */
template <> struct StageCfg<9> { static constexpr int SHM = 2; static constexpr bool SOFT = true;  static constexpr int BS = 256, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 9 with 320 threads (10 warps) per SM */
template <> struct StageCfg<10> { static constexpr int SHM = 2; static constexpr bool SOFT = true;  static constexpr int BS = 320, MINB = 1, REFILL = 16, PERIOD = 4; };
/* soft lockstep, one block of 192 threads per SM with history and LU in
   shared memory (fits with FP32 factors) */
template <> struct StageCfg<11> { static constexpr int SHM = 1; static constexpr bool SOFT = true;  static constexpr int BS = 192, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 9 with 384 threads (12 warps) per SM: the history of 384 cells fills
   the shared memory (221 KB for 12 species) */
template <> struct StageCfg<12> { static constexpr int SHM = 2; static constexpr bool SOFT = true;  static constexpr int BS = 384, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 8 (thread-local arrays, soft lockstep) in one block of 256 threads per
   SM (255 registers) or of 512 (128 registers): for networks above 32
   solver species, whose arrays live in local memory either way */
template <> struct StageCfg<15> { static constexpr int SHM = 0; static constexpr bool SOFT = true;  static constexpr int BS = 256, MINB = 1, REFILL = 16, PERIOD = 4; };
template <> struct StageCfg<16> { static constexpr int SHM = 0; static constexpr bool SOFT = true;  static constexpr int BS = 512, MINB = 1, REFILL = 16, PERIOD = 4; };
/* as 12, idle lanes refilled on every 32nd trip only (fewer, larger cell
   set-ups; measured on PRIMORDIAL's long solves: 1.6 % faster with FP32
   factors, 4.5 % slower in FP64; slower on short operator-split solves,
   whose lanes then wait longer for new cells) */
template <> struct StageCfg<17> { static constexpr int SHM = 2; static constexpr bool SOFT = true;  static constexpr int BS = 384, MINB = 1, REFILL = 32, PERIOD = 4; };
/* as 15 and 8 (soft lockstep, 256 or 384 threads) with the state vector y
   in shared memory (networks above 32 solver species; where blk_kernel.cuh
   covers the network, staging 18 is its kernel) */
template <> struct StageCfg<18> { static constexpr int SHM = 4; static constexpr bool SOFT = true;  static constexpr int BS = 256, MINB = 1, REFILL = 16, PERIOD = 4; };
template <> struct StageCfg<19> { static constexpr int SHM = 4; static constexpr bool SOFT = true;  static constexpr int BS = 384, MINB = 1, REFILL = 16, PERIOD = 4; };
/* staging 3's shape (three 128-thread blocks per SM, so that blocks of
   several solves share an SM) with the state vector in shared memory
   (networks above 32 solver species) */
template <> struct StageCfg<20> { static constexpr int SHM = 4; static constexpr bool SOFT = false; static constexpr int BS = 128, MINB = 3, REFILL = 16, PERIOD = 4; };
/* staging 3's shape with the history in shared memory and the block's four
   warps in soft lockstep (where three blocks' histories fit an SM: up to 12
   solver species) */
template <> struct StageCfg<21> { static constexpr int SHM = 2; static constexpr bool SOFT = true;  static constexpr int BS = 128, MINB = 3, REFILL = 16, PERIOD = 4; };

/* not a caller's choice: the shape of stagings 3 and 9 for few cells (see
   launch) -- as 2 with the block's four warps in soft lockstep */
constexpr int SPREAD_STAGE = 22;
template <> struct StageCfg<22> { static constexpr int SHM = 1; static constexpr bool SOFT = true;  static constexpr int BS = 128, MINB = 1, REFILL = 16, PERIOD = 4; };

/* Soft lockstep.  The warps of a block wait for each other at the top of
   every trip of the cell loop, so they run the same phase code at the same
   time and share instruction fetches.  No barrier instruction is used: lane
   0 of a warp counts itself in with a shared-memory atomic and polls a
   generation word, sleeping between polls, at most SOFT_SPIN_LIMIT times;
   after that it goes on alone.  Nothing a cell computes depends on the
   lockstep (every decision stays per lane or per warp), so a late, lost or
   early arrival costs time and never changes a result, and no wait is
   unbounded. */
struct SoftSync {
    unsigned arrive; /* warps counted in for the current generation */
    unsigned gen;    /* generation, bumped by the warp that completes it */
    unsigned active; /* warps still in the cell loop */
};
constexpr int SOFT_SPIN_LIMIT = 4096; /* polls of >= 64 ns: about 0.3 ms at most */

/* completes the current generation */
__device__ __forceinline__ void soft_release(SoftSync* s)
{
    atomicExch(&s->arrive, 0u);
    __threadfence_block();
    atomicAdd(&s->gen, 1u);
}

__device__ __forceinline__ void soft_sync(SoftSync* s, int lane)
{
    __syncwarp();
    if (lane == 0) {
        const unsigned g = *(volatile unsigned*)&s->gen;
        const unsigned n = atomicAdd(&s->arrive, 1u) + 1u;
        if (n >= *(volatile unsigned*)&s->active) {
            soft_release(s);
        } else {
            for (int i = 0; i < SOFT_SPIN_LIMIT; ++i) {
                if (*(volatile unsigned*)&s->gen != g)
                    break;
                __nanosleep(64);
            }
        }
    }
    __syncwarp();
}

/* a warp leaves the cell loop: if the others already wait for it, release them */
__device__ __forceinline__ void soft_leave(SoftSync* s, int lane)
{
    if (lane == 0) {
        const unsigned left = atomicSub(&s->active, 1u) - 1u;
        if (left > 0 && *(volatile unsigned*)&s->arrive >= left)
            soft_release(s);
    }
}


/* An FP64 LU with the correctly rounded reciprocals of its pivots beside it.
   A division by a pivot is then five dependent fused multiply-adds without a
   branch: the quotient from the reciprocal, corrected twice with its exact
   residual, which rounds correctly (P. Markstein, IBM J. Res. Dev. 34, 1990)
   up to the sign of zero: -0 by a positive pivot gives +0.  No result sees it:
   in the factors and solves a zero only adds and multiplies, and a correction
   is added to a sum that starts at +0.
   Operands for which that is not certain (far exponents, infinities, NaN, an
   all-ones significand) are recorded in bad, and the caller repeats the work
   with IEEE divisions.  The generated factorisation and solves pick these
   overloads of ov_pivot and ov_divp by the accessor's entry type. */
struct PivotRef {
    double* p;
    double* r;
    unsigned* bad;
    __device__ __forceinline__ operator double() const { return *p; }
    __device__ __forceinline__ void operator=(double v) const { *p = v; }
};

template <class Net, class A>
struct PivotLU {
    A a;       /* the packed factors */
    double* r; /* [ND] reciprocals, by pivot number */
    unsigned* bad;
    __device__ __forceinline__ PivotRef operator[](int i) const
    {
        const int k = Net::pivot_number(i);
        return PivotRef{&a[i], r + (k < 0 ? 0 : k), bad};
    }
};

template <class T>
__device__ __forceinline__ T ov_pivot(const PivotRef& p)
{
    const double v = p;
    const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu, lo = (unsigned)__double2loint(v);
    /* outside [2^-400, 2^400) or all ones below */
    *p.bad |= (hi - (623u << 20) >= (800u << 20)) | (lo == 0xffffffffu);
    *p.r = rcp_normal(v);
    return v;
}

template <class T>
__device__ __forceinline__ T ov_divp(T x, const PivotRef& p)
{
    const double d = p, r = *p.r;
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu, lo = (unsigned)__double2loint(x);
    /* outside [2^-500, 2^500) and not zero */
    *p.bad |= (hi - (523u << 20) >= (1000u << 20)) & ((hi | lo) != 0u);
    double q = x * r;
    q = __fma_rn(__fma_rn(-q, d, x), r, q);
    return __fma_rn(__fma_rn(-q, d, x), r, q);
}

template <class Net, class LUT, int SHM, int BS>
struct Staging;

template <class Net, class LUT, int BS>
struct Staging<Net, LUT, 0, BS> { /* thread-local arrays (registers / local memory) */
    using Hist = double (*)[Net::ND];
    using LU = LUT*;
    static constexpr size_t smem_bytes = 0;
};

template <class Net, class LUT, int BS>
struct Staging<Net, LUT, 1, BS> { /* shared memory, [entry][lane] */
    using Hist = LaneHist<Net::ND, BS>;
    using LU = LaneCol<LUT, BS>;
    static constexpr size_t hist_bytes = sizeof(double) * (MAXQ + 1) * Net::ND * BS;
    static constexpr size_t smem_bytes = hist_bytes + sizeof(LUT) * Net::NNZ * BS;
};

template <class Net, class LUT, int BS>
struct Staging<Net, LUT, 4, BS> { /* the state vector y in shared memory, history and LU thread-local */
    using Hist = double (*)[Net::ND];
    using LU = LUT*;
    /* one row of NEQ + 1 doubles per thread: the odd row length spreads a
       warp's accesses to one species over the banks */
    static constexpr int YROW = Net::NEQ + 1;
    static constexpr size_t smem_bytes = sizeof(double) * YROW * BS;
};

template <class Net, class LUT, int BS>
struct Staging<Net, LUT, 2, BS> { /* history in shared memory, LU thread-local */
    using Hist = LaneHist<Net::ND, BS>;
    using LU = LUT*;
    static constexpr size_t hist_bytes = sizeof(double) * (MAXQ + 1) * Net::ND * BS;
    static constexpr size_t smem_bytes = hist_bytes;
};

template <class Net, int G, class LUT, int SHM = 0, int BS = 128>
struct Cell {
    static constexpr int N = Net::NEQ;  /* full state */
    static constexpr int ND = Net::ND;  /* solver state */
    static constexpr int NF = Net::NF;
    static constexpr int NNZ = Net::NNZ;
    static constexpr int NR = Net::NREA > 0 ? Net::NREA : 1;
    static constexpr bool SCALED = sizeof(LUT) == 4;
    /* a small network's thread-local history is indexed by constants only,
       the columns beyond the order predicated off, so that it lives in
       registers.  With this, the reductions by words in lockstep groups, the
       exact quotient by the species count and PivotLU (below): ROBER, one
       lockstep group 0.54 -> 0.44 ms, 128 groups 0.60 -> 0.48 ms; OREGO,
       65,536 cells FP64 13.3 (staging 2) -> 12.4 ms (staging 3) */
    static constexpr bool REGH = ND <= 4 && SHM == 0;
    /* FP64 pivots with their reciprocals (PivotLU) for small networks, whose
       trip is a chain of dependent operations.  12 species: 175 against 145
       ms (PRIMORDIAL, 1,048,576 cells, FP64; the second copy of the code
       spills); with the reciprocals in the solves alone 146.  Not where the
       matrix keeps entries of the factorisation before, which must not be
       repeated. */
    static constexpr bool PIV = !SCALED && ND <= 4 && !Net::HC_FD;

    typename Staging<Net, LUT, SHM, BS>::Hist yns; /* Nordsieck history y_NS(0:5) */
    /* 16-byte aligned, so that neighbouring entries can move in one 128-bit
       access when the arrays live in local memory */
    alignas(16) double en[ND];
    alignas(16) double eno[ND];
    alignas(16) double w2[ND];
    /* the full state: a thread-local array, or (SHM 4) this thread's row in
       shared memory, which the network code reloads instead of spilling */
    alignas(16) std::conditional_t<SHM == 4, double*, double[N]> y;
    typename Staging<Net, LUT, SHM, BS>::LU a; /* packed LU of the iteration matrix */
    double* rp;                                /* PIV: reciprocals of its pivots */
    /* temperature part of the rates: an array of its own, not a member.  The
       set-up call that fills it takes its address, and as a member it would
       keep this whole object (state, weights, corrections, every control
       word) in local memory: PRIMORDIAL then executed 2.9 times the local
       loads and stores, and was 1.15 times slower (1,048,576 cells, FP32
       LU: 135.9 ms at its best shape, 118.1 ms without, one 256-thread
       block per SM; FP64 175.6 and 162.6 ms) */
    double* rT;
    /* FP32 LU: the scale of species j is 2^sce[j] (kept as an exponent, the
       factors are formed only while the Jacobian and the solve run) */
    short sce[SCALED ? ND : 1];

    double t, h, told, tstop, crate, jchg, cerr, tint;
    double fz_add; /* 0, or NaN when a frozen species has a non-finite error weight */
    int q, swu, lju, fet, fc, it, ss_mode, wait;
    bool ujac, nuo, first, msk, fz_neg;
    bool ieee; /* PIV: these factors need IEEE divisions */
    int status, attempts, steps, ltef, convf, newt, jacs, ppass;

    /* x / N for the full species count: for a power of two N the product
       by 2^-k, which rounds exactly as the division does (one rounding of
       the same exact value), without the division's instruction sequence */
    __device__ __forceinline__ static double div_n(double x)
    {
        if constexpr ((N & (N - 1)) == 0) {
            return x * (1.0 / N);
        } else {
            /* the quotient from the rounded reciprocal, corrected twice with
               its exact residual: correctly rounded (Markstein, as above)
               where nothing underflows or overflows */
            const double r = 1.0 / N;
            double v = x * r;
            v = __fma_rn(__fma_rn(-(double)N, v, x), r, v);
            v = __fma_rn(__fma_rn(-(double)N, v, x), r, v);
            if (x != 0.0 && (unsigned)__double2hiint(x) - (123u << 20) >= (1900u << 20))
                v = x / N;
            return v;
        }
    }

    /* WeightedNorm1 (src/odevec.F90:669-684) over the solver state; the
       lane's own sum of squares is left in s_lane */
    __device__ __forceinline__ double wnorm(const double* e, double& s_lane) const
    {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j)
            s = s + e[j] * e[j] * w2[j];
        s = s + fz_add;
        s_lane = s;
        double v = msk ? sqrt(div_n(s)) : -HUGE_VAL;
        return group_max<G>(v);
    }
    __device__ __forceinline__ double wnorm(const double* e) const
    {
        double s;
        return wnorm(e, s);
    }

    /* the square of wnorm(e): div_n of the sum of squares, before the root */
    __device__ __forceinline__ double wnorm_sq(const double* e) const
    {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j)
            s = s + e[j] * e[j] * w2[j];
        s = s + fz_add;
        return group_max<G>(msk ? div_n(s) : -HUGE_VAL);
    }

    /* the square of WeightedNorm2 of y_NS(:,:,col) for a runtime column */
    __device__ __forceinline__ double wnorm_ns_sq(int col) const
    {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            double e;
            if constexpr (REGH) {
                e = yns[1][j];
#pragma unroll
                for (int k = 2; k <= MAXQ; ++k)
                    e = k == col ? yns[k][j] : e;
            } else {
                e = yns[col][j];
            }
            s = s + e * e * w2[j];
        }
        s = s + fz_add;
        return group_max<G>(msk ? div_n(s) : -HUGE_VAL);
    }

    /* CalcErrorWeightInvSquared (src/odevec.F90:706-716).  Up to 16 species
       the reciprocals run without branches, side by side (a correctly rounded
       __drcp_rn is a branch each, so twelve ran one after another): PRIMORDIAL
       with FP32 factors 107.4 -> 102.9 ms, FP64 149.8 -> 144.5 ms
       (1,048,576 cells).  Above, the second copy of the code costs more than
       the chains (64 species: 474 against 498 ms). */
    __device__ __forceinline__ void weights(double rtol, double atol)
    {
        if constexpr (ND <= 16) {
            unsigned odd = 0;
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                const double x = rtol * fabs(y[Net::dyn(j)]) + atol;
                odd |= rcp_odd(x);
                const double w = rcp_normal(x);
                w2[j] = w * w;
            }
            if (!odd)
                return;
        }
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            /* correctly rounded reciprocal: the same bits as 1.0 / x */
            double w = __drcp_rn(rtol * fabs(y[Net::dyn(j)]) + atol);
            w2[j] = w * w;
        }
    }

    /* frozen species: constant state, so their weights and signs are fixed */
    __device__ __forceinline__ void frozen_flags(double rtol, double atol)
    {
        bool bad = false, neg = false;
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const double v = y[Net::frozen(j)];
            double w = 1.0 / (rtol * fabs(v) + atol);
            w = w * w;
            bad |= !(w - w == 0.0); /* inf or NaN */
            neg |= v < 0.0;
        }
        fz_add = bad ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        fz_neg = neg;
    }

    /* PredictSolution (src/odevec.F90:769-793): per species, the Pascal
       triangle y_NS(k-1) += y_NS(k) for l = 0..q-1, k = q..l+1, in the
       reference's order, on register copies of the history.  The history is
       indexed by runtime order only; species indices stay compile-time so
       en, w2 and y remain in registers. */
    __device__ __forceinline__ void predict()
    {
        ppass += q * (q + 1) / 2;
#pragma unroll 4
        for (int j = 0; j < ND; ++j) {
            double v[MAXQ + 1];
#pragma unroll
            for (int k = 0; k <= MAXQ; ++k)
                v[k] = yns[k][j];
#pragma unroll
            for (int l = 0; l < MAXQ; ++l)
#pragma unroll
                for (int k = MAXQ; k >= 1; --k)
                    if (l <= q - 1 && k <= q && k >= l + 1)
                        v[k - 1] = v[k] + v[k - 1];
#pragma unroll
            for (int k = 0; k < MAXQ; ++k)
                yns[k][j] = v[k];
        }
#pragma unroll
        for (int j = 0; j < ND; ++j)
            en[j] = 0.0;
    }

    /* ResetSystem (src/odevec.F90:526-544) */
    __device__ __forceinline__ void reset()
    {
        ppass += q * (q + 1) / 2;
#pragma unroll 4
        for (int j = 0; j < ND; ++j) {
            double v[MAXQ + 1];
#pragma unroll
            for (int k = 0; k <= MAXQ; ++k)
                v[k] = yns[k][j];
#pragma unroll
            for (int k = 0; k < MAXQ; ++k)
#pragma unroll
                for (int jj = MAXQ; jj >= 1; --jj)
                    if (k <= q - 1 && jj <= q && jj >= k + 1)
                        v[jj - 1] = v[jj - 1] - v[jj];
#pragma unroll
            for (int k = 0; k < MAXQ; ++k)
                yns[k][j] = v[k];
        }
    }

    /* SetStepSize (src/odevec.F90:720-743) */
    __device__ __forceinline__ void set_step(double dt_scale)
    {
        double dtt = 1.0;
        if constexpr (REGH) {
#pragma unroll
            for (int k = 1; k <= MAXQ; ++k) {
                dtt = dt_scale * dtt;
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    if (k <= q)
                        yns[k][j] = yns[k][j] * dtt;
            }
        } else {
#pragma unroll 1
            for (int k = 1; k <= q; ++k) {
                dtt = dt_scale * dtt;
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    yns[k][j] = yns[k][j] * dtt;
            }
        }
        h = h * dt_scale;
        jchg = jchg * dt_scale;
    }

    /* UpdateNordsieck (src/odevec.F90:747-765) */
    __device__ __forceinline__ void update_nordsieck()
    {
        if constexpr (REGH) {
#pragma unroll
            for (int k = 0; k <= MAXQ; ++k) {
                const double c = lcoef(q, k);
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    if (k <= q)
                        yns[k][j] = yns[k][j] + en[j] * c;
            }
        } else {
#pragma unroll 1
            for (int k = 0; k <= q; ++k) {
                const double c = lcoef(q, k);
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    yns[k][j] = yns[k][j] + en[j] * c;
            }
        }
    }

    /* CalcStepSizeOrder (src/odevec.F90:547-618); returns dt_scale */
    __device__ __forceinline__ double step_size_order()
    {
        const int order = q;
        const bool has_down = order != 1, has_up = !(order == MAXQ || nuo);
        /* squared norms; a lockstep group (uniform order) skips unused ones */
        const double x_down = G == 1 || has_down ? wnorm_ns_sq(order) : 0.0;
        const double x_same = wnorm_sq(en);
        double x_up = 0.0;
        if (G == 1 || has_up) {
            double d[ND];
#pragma unroll
            for (int j = 0; j < ND; ++j)
                d[j] = en[j] - eno[j];
            x_up = wnorm_sq(d);
        }
        int loc;
        bool big;
        double s = step_choice(order, has_down, has_up, x_down, x_same, x_up, loc, big);
        if (big) {
            if (loc == 1) {
                if (order != 1)
                    q = order - 1;
                else
                    status = OV_ERR_ORDER;
            } else if (loc == 3) {
                if (order != MAXQ) {
                    const double c = lcoef(order, order);
#pragma unroll
                    for (int j = 0; j < ND; ++j) {
                        const double v = c * en[j] / (order + 1.0);
                        if constexpr (REGH) {
#pragma unroll
                            for (int k = 2; k <= MAXQ; ++k)
                                yns[k][j] = k == order + 1 ? v : yns[k][j];
                        } else {
                            yns[order + 1][j] = v;
                        }
                    }
                    q = order + 1;
                } else
                    status = OV_ERR_ORDER;
            }
        }
        double upper;
        if (first) {
            upper = 1e4;
            first = false;
        } else
            upper = 10.0;
        s = upper < s ? upper : s;
        jchg = jchg * s;
        swu = 0;
        nuo = false;
        return s;
    }

    /* CheckConvergence (src/odevec.F90:622-665), den in d */
    __device__ __forceinline__ void check_convergence(const double* d, bool& failed, bool& converged)
    {
        double s_lane;
        const double err = wnorm(d, s_lane);
        double rate_tmp = 0.0;
        if (it != 0) {
            rate_tmp = err / cerr;
            crate = fmax(0.2 * crate, rate_tmp);
        }
        const double r15 = 1.5 * crate;
        const double crit = err * (1.0 < r15 ? 1.0 : r15);
        /* a NaN in den or in the weights (src/odevec.F90:645) makes its
           term and so the lane's sum of squares NaN: the entries are only
           scanned when that sum is NaN */
        bool nan = false;
        if (s_lane != s_lane) {
            nan = fz_add != fz_add;
#pragma unroll
            for (int j = 0; j < ND; ++j)
                nan |= (d[j] != d[j]) | (w2[j] != w2[j]);
        }
        if (group_any<G>(nan)) {
            failed = true;
            return;
        }
        /* crit / D < 1: the rounded quotient is below 1 exactly when crit < D */
        if (crit < conv_divisor(q)) {
            converged = true;
            return;
        }
        if (it >= 2 && crate > 2.0 * rate_tmp)
            failed = true;
        else if (it == 3)
            failed = true;
        else {
            failed = false;
            cerr = err;
            it = it + 1;
        }
    }

    __device__ __forceinline__ bool any_negative_yns0() const
    {
        bool neg = fz_neg;
#pragma unroll
        for (int j = 0; j < ND; ++j)
            neg |= yns[0][j] < 0.0;
        return group_any<G>(msk && neg);
    }

    __device__ __forceinline__ bool any_negative_y() const
    {
        bool neg = fz_neg;
#pragma unroll
        for (int j = 0; j < ND; ++j)
            neg |= y[Net::dyn(j)] < 0.0;
        return group_any<G>(msk && neg);
    }

    /* GetJac + LUDecompose (src/odevec.F90:301-315) */
    __device__ __forceinline__ void jacobian_lu()
    {
        double sc[SCALED ? ND : 1], isc[SCALED ? ND : 1];
        if constexpr (SCALED) {
            /* scale by powers of two close to the error weights (exact in
               FP64), then round to FP32 */
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                int e = (int)((ov_d2bits(w2[j]) >> 52) & 0x7ff) - 1023;
                int hexp = e >= 0 ? e / 2 : -((-e + 1) / 2);
                hexp = hexp > 480 ? 480 : (hexp < -480 ? -480 : hexp);
                sce[j] = (short)hexp;
                sc[j] = ov_pow2i(hexp);
                isc[j] = ov_pow2i(-hexp);
            }
        }
        ieee = false;
#pragma unroll 1
        for (;;) {
            if constexpr (Net::LU_METHOD == 3) {
                fd_jacobian(sc, isc);
            } else {
                double k[NR];
                Net::rates_k(y, rT, k);
                if constexpr (!SCALED)
                    Net::template jac<LUT>(y, k, lcoef(q, 0), h, a);
                else
                    Net::template jac_scaled<LUT>(y, k, lcoef(q, 0), h, a, sc, isc);
            }
            /* for LUmethod 2 jac() wrote the symbolic factors */
            if constexpr (PIV) {
                if (!ieee) {
                    unsigned bad = 0u;
                    Net::template lu_factor<LUT>(PivotLU<Net, decltype(a)>{a, rp, &bad});
                    /* once more from the matrix: the whole lockstep group,
                       whose difference quotients take a norm over the group
                       (the same values either way) */
                    if (group_any<G>(bad != 0u)) {
                        ieee = true;
                        continue;
                    }
                    break;
                }
            }
            Net::template lu_factor<LUT>(a);
            break;
        }
    }

    /* CalcJac_dense (src/odevec.F90:469-506), the DRPEPJ difference
       quotients: P(:,k) = -(dt*beta/r) * (f(y + r e_k) - f(y)), then 1 is
       added on the diagonal.  Only the solver-state columns are formed:
       the rows and columns of frozen species are those of the identity
       whatever their off-diagonal values, so they never reach a solution.
       Every array index is a compile-time constant (the perturbed column
       is selected, not indexed), so the state stays in registers. */
    __device__ __forceinline__ void fd_jacobian(const double* sc, const double* isc)
    {
        const double uround = 2.2204460492503131e-16;  /* 2^-52 */
        const double srur = 1.4901161193847656e-08;    /* 2^-26 */
        const double beta = lcoef(q, 0);
        double k[NR], f0[N];
        Net::rates_k(y, rT, k);
        Net::rhs(y, k, f0);
        double e[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j)
            e[j] = f0[Net::dyn(j)];
        const double fac = wnorm(e);
        double r0 = 1e3 * fabs(h) * uround * (double)N * fac;
        if (r0 == 0.0)
            r0 = 1.0;
#pragma unroll 1
        for (int col = 0; col < ND; ++col) {
            double yy[N];
            double yk = 0.0, wk = 0.0;
#pragma unroll
            for (int j = 0; j < N; ++j)
                yy[j] = y[j];
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                if (j == col) {
                    yk = y[Net::dyn(j)];
                    wk = w2[j];
                }
            }
            const double a1 = srur * fabs(yk), a2 = r0 / sqrt(wk);
            const double r = a1 >= a2 ? a1 : a2;
            const double fk = -(h * beta / r);
#pragma unroll
            for (int j = 0; j < ND; ++j)
                if (j == col)
                    yy[Net::dyn(j)] = yk + r;
            double k1[NR], f1[N];
            Net::rates_k(yy, rT, k1);
            Net::rhs(yy, k1, f1);
#pragma unroll
            for (int c = 0; c < ND; ++c) {
                if (c == col) {
#pragma unroll
                    for (int i = 0; i < ND; ++i) {
                        double v = (f1[Net::dyn(i)] - f0[Net::dyn(i)]) * fk;
                        if (i == c)
                            v = 1.0 + v;
                        if constexpr (SCALED)
                            a[Net::pidx(i, c)] = (LUT)(v * sc[i] * isc[c]);
                        else
                            a[Net::pidx(i, c)] = v;
                    }
                }
            }
        }
    }

    /* residual, solve, Newton update (src/odevec.F90:323-352) */
    __device__ __forceinline__ void newton_update(const double* f, double* den)
    {
        double res[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j)
            res[j] = h * f[Net::dyn(j)] - (yns[1][j] + en[j]);
        if constexpr (SCALED) {
            double sc[ND], isc[ND];
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                sc[j] = ov_pow2i(sce[j]);
                isc[j] = ov_pow2i(-sce[j]);
            }
            Net::template lu_solve<LUT>(a, res, den, sc, isc);
        } else if constexpr (PIV) {
            unsigned bad = ieee ? 1u : 0u;
            Net::template lu_solve<LUT>(PivotLU<Net, decltype(a)>{a, rp, &bad}, res, den, nullptr, nullptr);
            if (bad)
                Net::template lu_solve<LUT>(a, res, den, nullptr, nullptr);
        } else {
            Net::template lu_solve<LUT>(a, res, den, nullptr, nullptr);
        }
        const double l0 = lcoef(q, 0);
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            en[j] = en[j] + den[j];
            if (msk)
                y[Net::dyn(j)] = yns[0][j] + l0 * en[j];
        }
    }

    /* CalcInitialStepSize (src/odevec.F90:216-238), f holds f(y) */
    __device__ __forceinline__ double initial_step(const double* f, double rtol, double atol)
    {
        weights(rtol, atol);
        const double tol = rtol;
        const double W0 = fabs(t) > fabs(tstop) ? fabs(t) : fabs(tstop);
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            const double fj = f[Net::dyn(j)];
            s = s + fj * fj * (w2[j] * tol * tol);
        }
        s = s + fz_add;
        const double mx = group_max<G>(msk ? s : -HUGE_VAL);
        /* W0**(-2.0): a real exponent other than -1, 0, 1 or 2 is a pow() call
           in the reference's compiled Fortran, not 1/(W0*W0) */
        const double d = sqrt(tol / (ov_pow(W0, -2.0) + div_n(mx)));
        const double span = fabs(tstop - t);
        return d < span ? d : span;
    }

    /* InterpolateSolution (src/odevec.F90:998-1030) */
    __device__ __forceinline__ void interpolate()
    {
        const double rel_t = (tstop - t) / h;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            double acc;
            if constexpr (REGH) {
                acc = yns[MAXQ][j];
#pragma unroll
                for (int k = MAXQ - 1; k >= 0; --k) {
                    const double next = yns[k][j] + rel_t * acc;
                    acc = k < q ? next : yns[k][j];
                }
            } else {
                acc = yns[q][j];
#pragma unroll 1
                for (int k = q - 1; k >= 0; --k)
                    acc = yns[k][j] + rel_t * acc;
            }
            if (msk)
                y[Net::dyn(j)] = acc;
        }
    }

    /* end of an accepted step (src/odevec.F90:452-464, loop test :207) */
    __device__ __forceinline__ int finish_step(bool& write_y)
    {
        fet = 0;
        steps++;
        if (lju >= 20)
            ujac = true;
        else if (fabs(jchg - (double)1.0f) > (double)0.3f) /* 1.0 and 0.3 are single precision */
            ujac = true;
#pragma unroll
        for (int j = 0; j < ND; ++j)
            eno[j] = en[j];
        if (t < tstop) {
            told = t;
            return PH_PRED;
        }
        write_y = true;
        interpolate();
        tint = t;
        t = tstop;
        return PH_DONE;
    }

    /* resident workspace: [field][cell] with the launch's row stride */
    __device__ __forceinline__ void save_state(double* ws, int64_t n, int64_t cell) const
    {
        int f = 0;
#pragma unroll (REGH ? MAXQ + 1 : 1)
        for (int k = 0; k <= MAXQ; ++k)
#pragma unroll
            for (int j = 0; j < ND; ++j)
                ws[(f + k * ND + j) * n + cell] = yns[k][j];
        f += (MAXQ + 1) * ND;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            ws[(f + j) * n + cell] = eno[j];
            ws[(f + ND + j) * n + cell] = w2[j];
        }
        f += 2 * ND;
        const double sc[12] = {tint, h, crate, jchg, (double)q, (double)swu, (double)lju, (double)fet,
                               (double)fc, ujac ? 1.0 : 0.0, nuo ? 1.0 : 0.0, first ? 1.0 : 0.0};
#pragma unroll
        for (int i = 0; i < 12; ++i)
            ws[(f + i) * n + cell] = sc[i];
    }

    __device__ __forceinline__ void load_state(const double* ws, int64_t n, int64_t cell)
    {
        int f = 0;
#pragma unroll (REGH ? MAXQ + 1 : 1)
        for (int k = 0; k <= MAXQ; ++k)
#pragma unroll
            for (int j = 0; j < ND; ++j)
                yns[k][j] = ws[(f + k * ND + j) * n + cell];
        f += (MAXQ + 1) * ND;
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            eno[j] = ws[(f + j) * n + cell];
            w2[j] = ws[(f + ND + j) * n + cell];
        }
        f += 2 * ND;
        t = ws[(f + 0) * n + cell];
        h = ws[(f + 1) * n + cell];
        crate = ws[(f + 2) * n + cell];
        jchg = ws[(f + 3) * n + cell];
        q = (int)ws[(f + 4) * n + cell];
        swu = (int)ws[(f + 5) * n + cell];
        lju = (int)ws[(f + 6) * n + cell];
        fet = (int)ws[(f + 7) * n + cell];
        fc = (int)ws[(f + 8) * n + cell];
        ujac = ws[(f + 9) * n + cell] != 0.0;
        nuo = ws[(f + 10) * n + cell] != 0.0;
        first = ws[(f + 11) * n + cell] != 0.0;
    }
};

/* number of lanes of the warp for which b holds */
__device__ __forceinline__ int warp_count(bool b) { return __popc(__ballot_sync(FULL, b)); }


/* the temperature part of a cell's rates: from the launch's table, else
   evaluated here */
template <class Net>
__device__ __forceinline__ void cell_rates(const LaunchArgs& A, int64_t cell, double Tgas, double* r)
{
    if (A.rates) {
        const double* row = A.rates + cell * Net::NREA;
        if constexpr (Net::NREA % 2 == 0) {
            /* rows of an even number of doubles start on 16 bytes */
#pragma unroll
            for (int i = 0; i < Net::NREA; i += 2) {
                const double2 v = *reinterpret_cast<const double2*>(row + i);
                r[i] = v.x;
                r[i + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < Net::NREA; ++i)
                r[i] = row[i];
        }
    } else {
        Net::rates_T(Tgas, r);
    }
}

/* Fills the rate table of a launch, one thread per cell.  Bound by the FP64
   work of about forty exponentials, logarithms and powers, with every lane
   busy; in the solve kernel the same laws run for the two or three lanes of a
   warp that take a cell on the same trip, while the block's other warps wait.
   1,048,576 PRIMORDIAL cells: solve 116.0 -> 109.3 ms with FP32 factors,
   160.4 -> 152.3 ms in FP64, this kernel's time included. */
template <class Net>
__global__ void __launch_bounds__(128) rates_kernel(int64_t ncells, int64_t stride, const double* y, double* rates)
{
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncells;
         c += (int64_t)gridDim.x * blockDim.x) {
        alignas(16) double r[Net::NREA];
        Net::rates_T(y[(int64_t)Net::IDX_TGAS * stride + c], r);
        double* row = rates + c * Net::NREA;
        if constexpr (Net::NREA % 2 == 0) {
#pragma unroll
            for (int i = 0; i < Net::NREA; i += 2)
                *reinterpret_cast<double2*>(row + i) = make_double2(r[i], r[i + 1]);
        } else {
#pragma unroll
            for (int i = 0; i < Net::NREA; ++i)
                row[i] = r[i];
        }
    }
}

template <class Net>
cudaError_t launch_rates(const LaunchArgs& a, cudaStream_t stream)
{
    if constexpr (Net::NREA > 0) {
        const int64_t want = (a.ncells + 127) / 128;
        const int64_t most = 1 << 20; /* a grid-stride loop does the rest */
        rates_kernel<Net><<<(int)(want < most ? want : most), 128, 0, stream>>>(a.ncells, a.stride, a.y, a.rates);
        return cudaGetLastError();
    }
    return cudaErrorNotSupported;
}

/* The persistent cell loop of one network variant: the body of bdf_kernel,
   also run by the multi-network kernel for each of its jobs in turn.  A
   warp leaves it once the job's work counter has no cells left for it. */
template <class Net, int G, class LUT, int STAGE>
__device__ __forceinline__ void bdf_run(const LaunchArgs& A)
{
    constexpr int SHM = StageCfg<STAGE>::SHM;
    constexpr int BS = StageCfg<STAGE>::BS;
    using C = Cell<Net, G, LUT, SHM, BS>;
    constexpr int N = C::N;
    constexpr int ND = C::ND;
    const int lane = threadIdx.x & 31;
    const int64_t ncells = A.ncells;
    const int64_t stride = A.stride;
    if (A.run_if && *A.run_if == 0)
        return;

    C c;
    if constexpr (SHM == 4) {
        extern __shared__ __align__(16) unsigned char ov_smem[];
        c.y = reinterpret_cast<double*>(ov_smem) + (size_t)threadIdx.x * Staging<Net, LUT, 4, BS>::YROW;
    } else if constexpr (SHM != 0) {
        extern __shared__ __align__(16) unsigned char ov_smem[];
        c.yns = LaneHist<ND, BS>{reinterpret_cast<double*>(ov_smem) + threadIdx.x};
        if constexpr (SHM == 1)
            c.a = LaneCol<LUT, BS>{reinterpret_cast<LUT*>(ov_smem + Staging<Net, LUT, 1, BS>::hist_bytes)
                                   + threadIdx.x};
    }
    alignas(16) double history[(SHM == 0 || SHM == 4) ? MAXQ + 1 : 1][ND];
    alignas(16) LUT lu_local[SHM == 1 ? 1 : C::NNZ];
    if constexpr (SHM == 0 || SHM == 4)
        c.yns = history;
    if constexpr (SHM != 1) {
        c.a = lu_local;
        /* The LU of a network of more than a few species stays in memory:
           its constant indices would let the compiler spread it over
           registers that it does not have, and spill around every phase
           (PRIMORDIAL, 84 entries: 145 ms against 118 ms with FP32 factors,
           206 against 163 ms in FP64).  Taking its address in an empty
           statement keeps it an array.  The 506 FP32 factors of SYN64 are
           the exception (446 against 465 ms; its FP64 factors 576 against
           527 ms). */
        if constexpr (C::NNZ > 16 && (sizeof(LUT) == 8 || C::NNZ <= 128))
            asm volatile("" ::"l"(&lu_local[0]) : "memory");
    }
    double rcp_local[C::PIV ? ND : 1];
    c.rp = rcp_local;
    alignas(16) double rates_local[C::NR];
    c.rT = rates_local;
    int ph = G == 1 && A.lanes > 0 && lane >= A.lanes ? PH_EXHAUSTED : PH_IDLE;
    int64_t cell = -1;
    bool write_y = false;
    __shared__ SoftSync soft;
    if constexpr (StageCfg<STAGE>::SOFT) {
        if (threadIdx.x == 0) {
            soft.arrive = 0u;
            soft.gen = 0u;
            soft.active = blockDim.x / 32u;
        }
        __syncthreads(); /* at entry, with every thread converged */
    }

    /* A continued solve is a short one (a hydro step: some twelve steps a
       cell), whose lanes would wait half a REFILL period for new cells out of
       twenty trips: PRIMORDIAL, one step of 1,000,000 cells, refilled on every
       2nd / 4th / 8th / 16th trip 11.0 / 10.2 / 10.7 / 12.5 ms, 100,003 cells
       2.30 / 2.24 / 2.25 / 2.48 ms.  (Whole solves: 110.2 ms on every 8th,
       109.3 on every 16th.) */
    constexpr unsigned RESUME_REFILL = 4;
    const unsigned refill_mask = (A.resume == 1 ? RESUME_REFILL : StageCfg<STAGE>::REFILL) - 1u;
    unsigned trip = 0;
    for (;;) {
        /* ---- 1. idle lanes take new cells ---------------------------- */
        if (G == 1) {
            if constexpr (StageCfg<STAGE>::SOFT)
                soft_sync(&soft, lane);
            /* with REFILL > 1, idle lanes wait for every REFILL-th trip (the
               same trip in every warp of a lockstep block), so the costly
               cell set-up (loads, temperature rates, first right-hand side)
               runs for several lanes and warps at once instead of stretching
               trip after trip for one lane */
            const bool refill = StageCfg<STAGE>::REFILL <= 1 || (trip & refill_mask) == 0u;
            /* a yield request, seen on a refill trip after the first (so
               that every launch starts cells), turns the idle lanes into
               exhausted ones: the warp leaves once its running cells end */
            int stop = 0;
            if (refill && trip > 0u && A.yield) {
                if (lane == 0)
                    stop = *(volatile const int32_t*)A.yield;
                stop = __shfl_sync(FULL, stop, 0);
            }
            ++trip;
            if (stop && ph == PH_IDLE)
                ph = PH_EXHAUSTED;
            const unsigned need = refill && !stop ? __ballot_sync(FULL, ph == PH_IDLE) : 0u;
            if (need) {
                const int leader = __ffs(need) - 1;
                unsigned long long base = 0;
                if (lane == leader)
                    base = atomicAdd(A.queue, (unsigned long long)__popc(need));
                base = __shfl_sync(FULL, base, leader);
                if (ph == PH_IDLE) {
                    const int64_t q = (int64_t)(base + __popc(need & ((1u << lane) - 1u)));
                    if (q < ncells) {
                        cell = A.order ? (int64_t)A.order[q] : q;
                        ph = PH_START;
                    } else {
                        ph = PH_EXHAUSTED;
                    }
                }
            }
            if (__all_sync(FULL, ph == PH_EXHAUSTED)) {
                if constexpr (StageCfg<STAGE>::SOFT)
                    soft_leave(&soft, lane);
                break;
            }
        } else {
            if (ph == PH_IDLE) { /* warp-uniform */
                int stop = 0;
                if (trip > 0u && A.yield) { /* yield requests as above */
                    if (lane == 0)
                        stop = *(volatile const int32_t*)A.yield;
                    stop = __shfl_sync(FULL, stop, 0);
                }
                ++trip;
                if (stop) {
                    ph = PH_EXHAUSTED;
                } else {
                    unsigned long long g = 0;
                    if (lane == 0)
                        g = atomicAdd(A.queue, 1ull);
                    g = __shfl_sync(FULL, g, 0);
                    cell = (int64_t)g * 32 + lane;
                    ph = (int64_t)g * 32 < ncells ? PH_START : PH_EXHAUSTED;
                }
            }
            if (ph == PH_EXHAUSTED)
                break;
        }

        /* ---- load + SolveODE set-up (src/odevec.F90:169-198) --------- */
        if (ph == PH_START) {
#pragma unroll
            for (int j = 0; j < N; ++j)
                c.y[j] = A.y[(int64_t)j * stride + cell];
            c.t = A.t[cell];
            c.h = A.dt[cell];
            if (A.save_y) {
                /* the inputs, for the FP32-LU form's escalation */
#pragma unroll
                for (int j = 0; j < N; ++j)
                    A.save_y[(int64_t)j * ncells + cell] = c.y[j];
                A.save_t[cell] = c.t;
                A.save_dt[cell] = c.h;
            }
            c.tstop = A.t_stop[cell];
            c.msk = A.mask ? (A.mask[cell] != 0) : true;
            c.status = OV_OK;
            c.attempts = c.steps = c.ltef = c.convf = c.newt = c.jacs = c.ppass = 0;
            c.first = true;
            c.q = 1;
            c.swu = 0;
            c.crate = 0.7;
            c.jchg = 0.0;
            c.nuo = false;
            c.fet = 0;
            c.fc = 0;
            c.ujac = true;
            c.lju = 0;
            c.cerr = 0.0;
            c.it = 0;
            c.wait = 0;
            c.ss_mode = 0;
#pragma unroll
            for (int k = 0; k <= MAXQ; ++k)
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    c.yns[k][j] = 0.0;
#pragma unroll
            for (int j = 0; j < ND; ++j)
                c.eno[j] = 0.0;
            if constexpr (Net::HC_FD) {
                /* the heating/cooling Jacobian leaves entries of cells with a
                   non-positive species as the storage holds them: zero at
                   the start, as the reference's InitOdevec leaves its LU */
#pragma unroll
                for (int kk = 0; kk < C::NNZ; ++kk)
                    c.a[kk] = (LUT)0;
            }
            write_y = false;
            bool skip = !group_any<G>(c.msk);
            if (G == 32) {
                const bool bad = c.t != __shfl_sync(FULL, c.t, 0) || c.h != __shfl_sync(FULL, c.h, 0)
                                 || c.tstop != __shfl_sync(FULL, c.tstop, 0);
                if (__any_sync(FULL, bad)) {
                    c.status = OV_ERR_GROUP_MISMATCH;
                    ph = PH_DONE;
                }
            }
            if (ph == PH_START) {
                c.weights(A.rtol, A.atol);
                c.frozen_flags(A.rtol, A.atol);
                if (skip) {
                    c.t = c.tstop; /* src/odevec.F90:187-191 */
                    ph = PH_DONE;
                } else if (A.resume == 1) {
                    /* continuation: the saved history, step, order and
                       weights; the state is the saved y_NS(0); rates and
                       Jacobian are recomputed (the caller may have changed
                       the temperature) */
                    c.load_state(A.ws, stride, cell);
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        if (c.msk)
                            c.y[Net::dyn(j)] = c.yns[0][j];
                    if constexpr (Net::NREA > 0)
                        cell_rates<Net>(A, cell, c.y[Net::IDX_TGAS], c.rT);
                    c.ujac = true;
                    if (c.t < c.tstop) {
                        c.told = c.t;
                        ph = PH_PRED;
                    } else {
                        write_y = true;
                        c.interpolate();
                        c.tint = c.t;
                        c.t = c.tstop;
                        ph = PH_DONE;
                    }
                } else {
                    if (A.resume == 2) {
                        /* a fresh SolveODE that keeps the previous call's
                           last correction vector, as the reference's solver
                           object does (this%en_old is never reset) */
#pragma unroll
                        for (int j = 0; j < ND; ++j)
                            c.eno[j] = A.ws[((int64_t)(MAXQ + 1) * ND + j) * stride + cell];
                    }
                    if constexpr (Net::NREA > 0)
                        cell_rates<Net>(A, cell, c.y[Net::IDX_TGAS], c.rT);
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        c.yns[0][j] = c.y[Net::dyn(j)];
                }
            }
        }

        /* ---- 2. predictor attempt (src/odevec.F90:259-299) ----------- */
        if (ph == PH_PRED) {
            if (++c.attempts > A.max_attempts) {
                c.status = OV_ERR_MAX_STEPS;
                ph = PH_DONE;
            } else {
                c.t = c.t + c.h;
                c.predict();
                if (A.check_neg && c.any_negative_yns0()) {
                    c.t = c.told;
                    c.reset();
                    c.set_step(0.25);
                    if (c.h <= A.dt_min) {
                        c.status = OV_ERR_DTMIN_PREDICTOR;
                        ph = PH_DONE;
                    }
                    /* else: another predictor attempt on the next trip */
                } else {
                    if (c.msk) {
#pragma unroll
                        for (int j = 0; j < ND; ++j)
                            c.y[Net::dyn(j)] = c.yns[0][j];
                    }
                    c.it = 0;
                    ph = c.ujac ? PH_JACWAIT : PH_NEWTON;
                    c.wait = 0;
                }
            }
        }

        /* ---- 3. Jacobian + LU for the waiting lanes (:301-315) ------- */
        {
            bool run;
            if (G == 1) {
                const int waiting = warp_count(ph == PH_JACWAIT);
                const int moving = warp_count(ph == PH_NEWTON || ph == PH_START || ph == PH_RESTART);
                if constexpr (StageCfg<STAGE>::PERIOD > 1) {
                    /* trip was counted up at the top of this trip */
                    constexpr unsigned P = StageCfg<STAGE>::PERIOD;
                    run = waiting > 0 && (trip % P == 1u % P || moving == 0);
                } else {
                    const bool aged = __any_sync(FULL, ph == PH_JACWAIT && c.wait >= A.max_wait);
                    run = waiting > 0 && (waiting >= A.jac_batch || moving == 0 || aged);
                }
            } else {
                run = ph == PH_JACWAIT;
            }
            if (run && ph == PH_JACWAIT) {
                c.jacobian_lu();
                c.jacs++;
                c.ujac = false;
                c.lju = 0;
                c.crate = 0.7;
                c.jchg = 1.0;
                ph = PH_NEWTON;
            } else if (ph == PH_JACWAIT) {
                c.wait++;
            }
        }

        /* ---- 4. right-hand side ------------------------------------- */
        double f[N];
        if (ph == PH_START || ph == PH_NEWTON || ph == PH_RESTART) {
            double k[C::NR];
            Net::rates_k(c.y, c.rT, k);
            Net::rhs(c.y, k, f);
        }

        /* ---- 5. consume it ------------------------------------------ */
        if (ph == PH_START) {
            /* src/odevec.F90:201-210 */
#pragma unroll
            for (int j = 0; j < ND; ++j)
                c.yns[1][j] = c.h * f[Net::dyn(j)];
            c.h = c.initial_step(f, A.rtol, A.atol);
            if (c.t < c.tstop) {
                c.told = c.t;
                ph = PH_PRED;
            } else {
                write_y = true;
                c.interpolate();
                c.tint = c.t;
                c.t = c.tstop;
                ph = PH_DONE;
            }
        } else if (ph == PH_RESTART) {
            /* src/odevec.F90:417-421 */
#pragma unroll
            for (int j = 0; j < ND; ++j)
                c.yns[1][j] = c.h * f[Net::dyn(j)];
            c.ujac = true;
            c.ss_mode = SS_RESTART;
            c.wait = 0;
            ph = PH_SSWAIT;
        } else if (ph == PH_NEWTON) {
            c.newt++;
            double den[ND];
            c.newton_update(f, den);
            bool failed = false, converged = false;
            c.check_convergence(den, failed, converged);
            if (A.check_neg && c.any_negative_y()) {
                failed = true;
                converged = false;
            }
            if (failed && !converged) {
                /* src/odevec.F90:375-393 */
                c.t = c.told;
                c.fc++;
                c.convf++;
                if (c.fc > 10) {
                    c.status = OV_ERR_CONV_FAILURES;
                    ph = PH_DONE;
                } else {
                    c.it = 0;
                    c.reset();
                    c.set_step(0.25);
                    if (c.h < A.dt_min) {
                        c.status = OV_ERR_DTMIN_CONV;
                        ph = PH_DONE;
                    } else {
                        c.ujac = true;
                        ph = PH_PRED;
                    }
                }
            } else if (converged) {
                c.fc = 0;
                /* local truncation error test (src/odevec.F90:400-455) */
                const bool lte = c.wnorm_sq(c.en) >= c_lte[c.q];
                c.weights(A.rtol, A.atol);
                if (lte) {
                    c.ltef++;
                    c.t = c.told;
                    if (c.fet >= 3) {
                        if (A.fix_restart)
                            c.reset();
                        c.q = 1;
                        if (c.msk) {
#pragma unroll
                            for (int j = 0; j < ND; ++j)
                                c.y[Net::dyn(j)] = c.yns[0][j];
                        }
                        ph = PH_RESTART;
                    } else {
                        c.reset();
                        c.ujac = true;
                        c.swu = 0;
                        c.nuo = true;
                        c.ss_mode = SS_REJECT;
                        c.wait = 0;
                        ph = PH_SSWAIT;
                    }
                } else {
                    c.swu++;
                    c.lju++;
                    c.update_nordsieck();
                    if (c.swu == c.q + 1) {
                        c.ss_mode = SS_ACCEPT;
                        c.wait = 0;
                        ph = PH_SSWAIT;
                    } else {
                        ph = c.finish_step(write_y);
                    }
                }
            }
            /* else: next Newton iteration on the next trip */
        }

        /* ---- 6. step-size / order selection for the waiting lanes --- */
        {
            bool run;
            if (G == 1) {
                const int waiting = warp_count(ph == PH_SSWAIT);
                const int moving = warp_count(ph == PH_PRED || ph == PH_NEWTON || ph == PH_RESTART);
                if constexpr (StageCfg<STAGE>::PERIOD > 1) {
                    run = waiting > 0 && (trip % StageCfg<STAGE>::PERIOD == 0u || moving == 0);
                } else {
                    const bool aged = __any_sync(FULL, ph == PH_SSWAIT && c.wait >= A.max_wait);
                    run = waiting > 0 && (waiting >= A.ss_batch || moving == 0 || aged);
                }
            } else {
                run = ph == PH_SSWAIT;
            }
            if (run && ph == PH_SSWAIT) {
                const double s = c.step_size_order();
                if (c.status) {
                    ph = PH_DONE;
                } else {
                    c.set_step(s);
                    if (c.ss_mode == SS_ACCEPT) {
                        ph = c.finish_step(write_y);
                    } else {
                        c.fet++; /* src/odevec.F90:434-439 */
                        ph = PH_PRED;
                    }
                }
            } else if (ph == PH_SSWAIT) {
                c.wait++;
            }
        }

        /* ---- 7. store finished cells -------------------------------- */
        if (ph == PH_DONE) {
            const bool ok = c.status == OV_OK;
            if (A.ws && ok && write_y)
                c.save_state(A.ws, stride, cell);
            if ((!ok || write_y) && c.msk) {
#pragma unroll
                for (int j = 0; j < ND; ++j)
                    A.y[(int64_t)Net::dyn(j) * stride + cell] = c.y[Net::dyn(j)];
            }
            A.t[cell] = c.t;
            if (c.status != OV_ERR_GROUP_MISMATCH)
                A.dt[cell] = c.h;
            if (A.status)
                A.status[cell] = c.status;
            if (A.stats) {
                int32_t* s = A.stats + cell * OV_NSTATS;
                s[0] = c.steps;
                s[1] = c.attempts;
                s[2] = c.ltef;
                s[3] = c.convf;
                s[4] = c.newt;
                s[5] = c.jacs;
                s[6] = c.q;
                s[7] = c.ppass;
            }
            ph = PH_IDLE;
        }
    }
}

template <class Net, int G, class LUT, int STAGE>
__global__ void __launch_bounds__(StageCfg<STAGE>::BS, StageCfg<STAGE>::MINB)
    bdf_kernel(const __grid_constant__ LaunchArgs A)
{
    bdf_run<Net, G, LUT, STAGE>(A);
}

/* warps per SM of a launch of few cells: one per scheduler */
constexpr int SPREAD_WARPS = 4;

template <class Net, int G, class LUT, int STAGE>
cudaError_t launch(const LaunchArgs& a, int block, int grid, cudaStream_t stream)
{
    using Cfg = StageCfg<STAGE>;
    auto kern = bdf_kernel<Net, G, LUT, STAGE>;
    constexpr size_t smem = Staging<Net, LUT, Cfg::SHM, Cfg::BS>::smem_bytes;
    const bool chosen = block > 0 || grid > 0; /* the caller fixes the shape */
    if (Cfg::SHM || block <= 0 || block > Cfg::BS)
        block = Cfg::BS;
    int sms = 0;
    cudaError_t err = device_sms(&sms);
    if (err != cudaSuccess)
        return err;
    LaunchArgs b = a;
    if constexpr (G == 1 && (STAGE == 3 || STAGE == 9) && Net::ND > 4 && Net::ND <= 32 &&
                  Staging<Net, LUT, 1, StageCfg<SPREAD_STAGE>::BS>::smem_bytes <= 226 * 1024) {
        /* Up to a few cells per lane of four warps per SM, the factors go into
           shared memory beside the history: with four warps they fit, and a
           trip then reads nothing but on-chip memory.  PRIMORDIAL, against
           staging 9: FP64 1,000 cells 7.0 -> 5.6 ms, 8,192 cells 10.3 -> 8.0,
           18,944 cells 11.2 -> 8.7, 32,000 cells 13.7 -> 10.6, 75,776 cells
           16.0 -> 15.6, 100,003 cells 18.9 -> 19.6; FP32-LU 1,000 cells 4.9 ->
           4.4 ms, 18,944 cells 7.1 -> 6.8, 56,832 cells 10.3 -> 9.9, 75,776
           cells 11.1 -> 12.2.  So the line lies at 4 cells per lane in FP64
           and 3 with FP32 factors.  Continued solves are short and gain more
           from a lane's shorter trip: 8 in FP64 (one step with contraction,
           100,003 cells 2.23 -> 1.99 ms, 150,001 cells 2.67 -> 2.46, 1,000,000
           cells equal).  Without the lockstep 8,192 cells take 8.5 instead of
           8.0 ms, 18,000 cells 9.8 instead of 8.4.  Up to four species the
           history is in registers instead. */
        const int64_t lanes = (int64_t)sms * SPREAD_WARPS * 32;
        const int per_lane = sizeof(LUT) == 8 ? (a.resume == 1 ? 8 : 4) : 3;
        if (!chosen && a.ncells <= lanes * per_lane)
            return launch<Net, G, LUT, SPREAD_STAGE>(a, 0, 0, stream);
    }
    /* only now, since a question about a kernel loads it: a process of small
       solves loads the one kernel that it runs */
    err = allow_smem((const void*)kern, smem);
    if (err != cudaSuccess)
        return err;
    if (Net::ND <= 32 && !chosen && a.ncells <= (int64_t)sms * SPREAD_WARPS * 32) {
        /* Few cells: over all SMs, at most one warp per scheduler and only as
           many lanes per warp as that takes.  The time is that of the longest
           cells' chain of steps then, and a warp's trip is the shorter the
           fewer cells share it and the fewer warps share its scheduler.
           PRIMORDIAL with FP32 factors, in blocks of 256 cells one after the
           other / four warps per SM / eight warps per SM: 1,000 cells 8.4 /
           4.6 / 5.4 ms, 4,096 cells 8.9 / 6.1 / 6.7, 8,192 cells 8.7 / 6.4 /
           7.7, 16,384 cells 9.2 / 7.5 / 8.4; from 32,768 cells on full warps
           are as fast or faster (9.4 against 9.8).  Not for large networks,
           whose warps live from sharing instruction fetches (SYN64 FP64, 3,001
           cells: 186 ms spread, 168 ms in 256-cell blocks). */
        int64_t groups, lanes = 1; /* work items: cells, or lockstep groups (a warp each) */
        groups = G == 1 ? a.ncells : (a.ncells + 31) / 32;
        int64_t warps = (groups + sms - 1) / sms; /* per SM */
        const int64_t most = Cfg::BS / 32 < SPREAD_WARPS ? Cfg::BS / 32 : SPREAD_WARPS;
        if (warps > most)
            warps = most;
        if (G == 1)
            lanes = (groups + sms * warps - 1) / (sms * warps);
        b.lanes = (int32_t)(lanes < 32 ? lanes : 32);
        block = (int)(32 * warps);
        const int64_t per_block = warps * (G == 1 ? (int64_t)b.lanes : 1);
        grid = (int)((groups + per_block - 1) / per_block);
        if (grid < 1)
            grid = 1;
    } else if (grid <= 0) {
        static Residency residency;
        err = resident_blocks(residency, (const void*)kern, block, smem, &grid);
        if (err != cudaSuccess)
            return err;
        const int64_t warps_needed = (a.ncells + 31) / 32;
        const int64_t blocks_needed = (warps_needed * 32 + block - 1) / block;
        if (blocks_needed < grid)
            grid = (int)blocks_needed;
        if (grid < 1)
            grid = 1;
    }
    kern<<<grid, block, smem, stream>>>(b);
    return cudaGetLastError();
}

/* shared-memory staging is compiled for per-cell control when the per-lane
   arrays of a block fit in 200 KB */
template <class Net, class LUT, int BS>
constexpr bool shm_fits()
{
    return Staging<Net, LUT, 1, BS>::smem_bytes <= 200 * 1024;
}

/* the same for the history alone */
template <class Net, int BS>
constexpr bool hist_fits()
{
    return Staging<Net, double, 2, BS>::smem_bytes <= 200 * 1024;
}

/* the histories of three blocks of 128 within an SM's shared memory */
template <class Net>
constexpr bool hist_fits_3x128()
{
    return 3 * (Staging<Net, double, 2, 128>::smem_bytes + 1024) <= 228 * 1024;
}

/* the state vectors of a block within the 227 KB a block may hold */
template <class Net, int BS>
constexpr bool y_fits()
{
    return Staging<Net, double, 4, BS>::smem_bytes <= 226 * 1024;
}

/* the history alone within the 227 KB a block may hold (less the soft
   lockstep words) */
template <class Net, int BS>
constexpr bool hist_fits_max()
{
    return Staging<Net, double, 2, BS>::smem_bytes <= 226 * 1024;
}

}  // namespace OV_MODE_NS
}  // namespace ov

#include "blk_kernel.cuh"
#include "wpc_kernel.cuh"

namespace ov {
namespace OV_MODE_NS {

/* ---- several networks in one launch ---------------------------------- */
/* One block of 256 threads per SM with all the registers of a thread.  A job
   runs as its network runs best alone: a large network as one block per 32
   cells (blk_kernel.cuh), another as staging 9 (soft lockstep, the history in
   shared memory) or, where a history does not fit, staging 15.  A large
   network's cells, which take longest, get their blocks first, the rest are
   shared out in proportion to cells times LU entries, an estimate of the
   jobs' work; a block whose job has no cells left takes cells of the others.
   16,384 ROBER, 65,536 PRIMORDIAL and 4,096 SYN64 cells, FP32-LU / FP64: 196 /
   254 ms with every network on one 384-thread block per SM and shares by cells
   alone, 40 / 60 ms so (46 with FP32-LU before the large network came first);
   65,536, 262,144 and 16,384 cells: 303 / 415 and 131 / 213 ms. */
template <class Net, class LUT, bool MANY>
struct MultiJob {
    static constexpr int STAGE = hist_fits<Net, 256>() ? 9 : 15;
    static constexpr bool BLOCK = blk_ok<Net, LUT>();
    /* a kernel for launches with many cells of it: a thread per cell for those
       (blk_split_cells) */
    static constexpr bool SPLIT = MANY && BLOCK && BLK_SPLIT && y_fits<Net, BLK_SPLIT_THREADS>();
    static constexpr size_t smem()
    {
        if constexpr (SPLIT) {
            constexpr size_t a = BlkLayout<Net, LUT>::smem_bytes;
            constexpr size_t b = Staging<Net, LUT, StageCfg<18>::SHM, StageCfg<18>::BS>::smem_bytes;
            return a > b ? a : b;
        } else if constexpr (BLOCK) {
            return BlkLayout<Net, LUT>::smem_bytes;
        } else {
            return Staging<Net, LUT, StageCfg<STAGE>::SHM, StageCfg<STAGE>::BS>::smem_bytes;
        }
    }
    __device__ __forceinline__ static void run(const LaunchArgs& A, bool many)
    {
        if constexpr (SPLIT) {
            if (many)
                bdf_run<Net, 1, LUT, 18>(A);
            else
                blk_run<Net, LUT>(A);
        } else if constexpr (BLOCK) {
            blk_run<Net, LUT>(A);
        } else {
            bdf_run<Net, 1, LUT, STAGE>(A);
        }
    }
};
constexpr int MULTI_BS = 256;
static_assert(32 * BLK_WARPS == MULTI_BS && StageCfg<9>::BS == MULTI_BS && StageCfg<15>::BS == MULTI_BS &&
                  StageCfg<18>::BS == MULTI_BS && StageCfg<9>::SOFT && StageCfg<15>::SOFT && StageCfg<18>::SOFT,
              "the jobs of a multi-network launch share one block shape and start with a barrier");

template <class LUT, bool MANY, class... Nets>
constexpr size_t multi_smem_bytes()
{
    size_t m = 0;
    ((m = MultiJob<Nets, LUT, MANY>::smem() > m ? MultiJob<Nets, LUT, MANY>::smem() : m), ...);
    return m;
}

template <class LUT, bool MANY, class... Nets>
struct MultiDispatch {
    __device__ __forceinline__ static void run(int, const LaunchArgs&, bool) {}
};
template <class LUT, bool MANY, class Net0, class... Rest>
struct MultiDispatch<LUT, MANY, Net0, Rest...> {
    __device__ __forceinline__ static void run(int idx, const LaunchArgs& A, bool many)
    {
        if (idx == 0)
            MultiJob<Net0, LUT, MANY>::run(A, many);
        else
            MultiDispatch<LUT, MANY, Rest...>::run(idx - 1, A, many);
    }
};

template <class LUT, bool MANY, class... Nets>
__global__ void __launch_bounds__(MULTI_BS, 1) bdf_multi_kernel(const __grid_constant__ MultiArgs P)
{
    int first = 0;
    while (first + 1 < P.njobs && (int)blockIdx.x >= P.block_start[first + 1])
        ++first;
    for (int k = 0; k < P.njobs; ++k) {
        const int j = (first + k) % P.njobs;
        MultiDispatch<LUT, MANY, Nets...>::run(P.net[j], P.job[j], P.many[j] != 0);
        /* a warp that leaves a job's loop first must not set up the lockstep
           words of the next job, if of the same network, while others use them
           (two jobs of 65,536 PRIMORDIAL cells, FP32-LU: 166-191 ms, 20 so; in
           front of the set-up the barrier costs a third of the speed) */
        __syncthreads();
    }
}

/* Launches the multi-network kernel on P (block ranges filled in here in
   proportion to the jobs' work, at least one block per job). */
template <class LUT, bool MANY, class... Nets>
cudaError_t launch_multi_kernel(MultiArgs& P, cudaStream_t stream)
{
    auto kern = bdf_multi_kernel<LUT, MANY, Nets...>;
    constexpr size_t smem = multi_smem_bytes<LUT, MANY, Nets...>();
    static_assert(smem <= 226 * 1024, "the set's largest state vectors exceed a block's shared memory");
    static Residency residency;
    int resident = 0;
    cudaError_t err = allow_smem((const void*)kern, smem);
    if (err == cudaSuccess)
        err = resident_blocks(residency, (const void*)kern, MULTI_BS, smem, &resident);
    if (err != cudaSuccess)
        return err;
    const int nnz[] = {Nets::NNZ...};
    const bool block[] = {MultiJob<Nets, LUT, MANY>::BLOCK...};
    /* Blocks of each job: first a block per 32 cells for the large networks
       (all but one per other job at most), whose cells take longest from
       start to end; the rest in proportion to cells times LU entries, an
       estimate of the work.  At least one per job. */
    int nb[MULTI_MAX_JOBS];
    int left = resident;
    double total = 0.0;
    for (int j = 0; j < P.njobs; ++j) {
        nb[j] = 1;
        --left;
        if (!block[P.net[j]])
            total += (double)P.job[j].ncells * nnz[P.net[j]];
    }
    for (int j = 0; j < P.njobs && left > 0; ++j)
        if (block[P.net[j]]) {
            const int64_t want = (P.job[j].ncells + 31) / 32 - 1;
            const int more = (int)(want < left ? want : left);
            if (more > 0) {
                nb[j] += more;
                left -= more;
            }
        }
    for (int j = 0; j < P.njobs && left > 0; ++j)
        if (!block[P.net[j]] && total > 0.0)
            nb[j] += (int)(left * ((double)P.job[j].ncells * nnz[P.net[j]]) / total);
    int start = 0;
    for (int j = 0; j < P.njobs; ++j) {
        P.block_start[j] = start;
        start += nb[j];
    }
    P.block_start[P.njobs] = start;
    kern<<<start, MULTI_BS, smem, stream>>>(P);
    return cudaGetLastError();
}

/* The thread-per-cell body of a large network is in a kernel of its own, for
   the launches that use it: beside it the compiler gives the other networks'
   bodies less (131,072 PRIMORDIAL cells, FP64: 32.0 ms without, 39.3 with).
   65,536 ROBER, 262,144 PRIMORDIAL and 262,144 SYN64 cells, FP64: 2,351 ms
   with SYN64 in the block kernel, 2,036 so. */
template <class LUT, class... Nets>
cudaError_t launch_multi(MultiArgs& P, cudaStream_t stream)
{
    if constexpr ((MultiJob<Nets, LUT, true>::SPLIT || ...)) {
        const bool split[] = {MultiJob<Nets, LUT, true>::SPLIT...};
        int sms = 0;
        const cudaError_t err = device_sms(&sms);
        if (err != cudaSuccess)
            return err;
        bool any = false;
        for (int j = 0; j < P.njobs; ++j) {
            P.many[j] = split[P.net[j]] && P.job[j].ncells >= blk_split_cells(sms);
            any = any || P.many[j];
        }
        if (any)
            return launch_multi_kernel<LUT, true, Nets...>(P, stream);
    }
    return launch_multi_kernel<LUT, false, Nets...>(P, stream);
}

}  // namespace OV_MODE_NS
}  // namespace ov

/* Defines the launcher of one network variant in the current mode.
   stage: 1 = thread-local arrays, 2 blocks of 128 per SM; 2 = history and
   LU in shared memory, 1 block of 128; 3, 4 = thread-local, 3 or 4 blocks of
   128 (fewer registers, more warps); 5 = shared memory, 1 block of 192;
   6 = thread-local, 1 block of 384; 7 = one warp per cell (wpc_kernel.cuh;
   constant-coefficient CSC variants); 8 = as 6 in soft lockstep; 9, 10 =
   soft lockstep in one block of 256 or 320 with the history in shared
   memory; 11 = soft lockstep in one block of 192 with history and LU in
   shared memory (where they fit); 12 = as 9 in one block of 384; 13, 14 =
   16 or 8 lanes per cell (wpc_kernel.cuh, as 7); 15, 16 = as 8 in one block
   of 256 or 512 (networks above 32 solver species); 17 = as 12 refilling on
   every 32nd trip; 18, 19 = as 8 in one block of 256 or 384 with the state
   vector in shared memory, 20 = as 3 with the state vector in shared memory
   (18-20: networks above 32 solver species; 18 is the block-per-32-cells
   kernel of blk_kernel.cuh for the networks that it covers); 21 = as 3 with the history in
   shared memory and the block in soft lockstep (up to 12 solver species).  With per-cell control stagings 2-6 and 8-16 refill idle
   lanes on every 16th trip, 17 on every 32nd, staging 1 on every trip.
   Stages 2-21 exist for per-cell control (G = 1). */
#define OV_STAGE_CASE(NET, LU, ST)                                                               \
    if (stage == ST)                                                                             \
        return launch<NET, 1, LU, ST>(a, block, grid, s);

/* Defines the multi-network launcher of one set of variants in the current
   mode: launch_multi_<sid>(P, lu, stream), lu 0 = FP64 LU, 1 = FP32 LU (fma
   mode only). */
#define OV_DEFINE_MULTI(sid, FP32, ...)                                                          \
    namespace ov {                                                                               \
    namespace OV_MODE_NS {                                                                       \
    cudaError_t launch_multi_##sid(MultiArgs& P, int lu, cudaStream_t s)                          \
    {                                                                                            \
        if (lu == 0)                                                                             \
            return launch_multi<double, __VA_ARGS__>(P, s);                                      \
        if constexpr (FP32) {                                                                    \
            if (lu == 1)                                                                         \
                return launch_multi<float, __VA_ARGS__>(P, s);                                   \
        }                                                                                        \
        return cudaErrorNotSupported;                                                            \
    }                                                                                            \
    }                                                                                            \
    }

#define OV_DEFINE_LAUNCHER(cid, FP32)                                                            \
    namespace ov {                                                                               \
    namespace OV_MODE_NS {                                                                       \
    cudaError_t launch_##cid(const LaunchArgs& a, int G, int lu, int stage, int block, int grid,  \
                             cudaStream_t s)                                                     \
    {                                                                                            \
        using NET = ov_net_##cid;                                                                \
        if (stage == STAGE_RATES)                                                                \
            return launch_rates<NET>(a, s);                                                      \
        if (G == 1 && lu == 0) {                                                                 \
            OV_STAGE_CASE(NET, double, 1)                                                        \
            OV_STAGE_CASE(NET, double, 3)                                                        \
            OV_STAGE_CASE(NET, double, 4)                                                        \
            OV_STAGE_CASE(NET, double, 6)                                                        \
            OV_STAGE_CASE(NET, double, 8)                                                        \
            if constexpr (NET::ND > 32) {                                                    \
                OV_STAGE_CASE(NET, double, 15)                                               \
                OV_STAGE_CASE(NET, double, 16)                                               \
                if constexpr (blk_ok<NET, double>()) {                                       \
                    if constexpr (BLK_SPLIT && y_fits<NET, 256>()) {                         \
                        int sms = 0;                                                         \
                        if (stage == 18 && device_sms(&sms) == cudaSuccess &&                \
                            a.ncells >= blk_split_cells(sms)) {                              \
                            OV_STAGE_CASE(NET, double, 18)                                   \
                        }                                                                    \
                    }                                                                        \
                    if (stage == 18)                                                         \
                        return launch_blk<NET, double>(a, grid, s);                          \
                } else if constexpr (y_fits<NET, 256>()) {                                   \
                    OV_STAGE_CASE(NET, double, 18)                                           \
                }                                                                            \
                if constexpr (y_fits<NET, 128>()) {                                          \
                    OV_STAGE_CASE(NET, double, 20)                                           \
                }                                                                            \
                if constexpr (y_fits<NET, 384>()) {                                          \
                    OV_STAGE_CASE(NET, double, 19)                                           \
                }                                                                            \
            }                                                                                \
            if constexpr (hist_fits_3x128<NET>()) {                                          \
                OV_STAGE_CASE(NET, double, 21)                                               \
            }                                                                                \
            if constexpr (hist_fits<NET, 256>()) {                                               \
                OV_STAGE_CASE(NET, double, 9)                                                    \
            }                                                                                    \
            if constexpr (hist_fits<NET, 320>()) {                                               \
                OV_STAGE_CASE(NET, double, 10)                                                   \
            }                                                                                    \
            if constexpr (hist_fits_max<NET, 384>()) {                                           \
                OV_STAGE_CASE(NET, double, 12)                                                   \
                OV_STAGE_CASE(NET, double, 17)                                               \
            }                                                                                    \
            if constexpr (shm_fits<NET, double, 192>()) {                                        \
                OV_STAGE_CASE(NET, double, 11)                                                   \
            }                                                                                    \
            if constexpr (wpc_ok<NET, double, 32>()) {                                       \
                if (stage == 7)                                                              \
                    return launch_wpc<NET, double, 32>(a, grid, s);                          \
            }                                                                                \
            if constexpr (wpc_ok<NET, double, 16>()) {                                       \
                if (stage == 13)                                                             \
                    return launch_wpc<NET, double, 16>(a, grid, s);                          \
            }                                                                                \
            if constexpr (wpc_ok<NET, double, 8>()) {                                        \
                if (stage == 14)                                                             \
                    return launch_wpc<NET, double, 8>(a, grid, s);                           \
            }                                                                                \
            if constexpr (shm_fits<NET, double, 128>()) {                                        \
                OV_STAGE_CASE(NET, double, 2)                                                    \
            }                                                                                    \
            return cudaErrorNotSupported;                                                        \
        }                                                                                        \
        if constexpr (FP32) {                                                                    \
            if (G == 1 && lu == 1) {                                                             \
                OV_STAGE_CASE(NET, float, 1)                                                     \
                OV_STAGE_CASE(NET, float, 3)                                                     \
                OV_STAGE_CASE(NET, float, 4)                                                     \
                OV_STAGE_CASE(NET, float, 6)                                                     \
                OV_STAGE_CASE(NET, float, 8)                                                     \
                if constexpr (NET::ND > 32) {                                                \
                    OV_STAGE_CASE(NET, float, 15)                                            \
                    OV_STAGE_CASE(NET, float, 16)                                            \
                    if constexpr (blk_ok<NET, float>()) {                                    \
                        if (stage == 18)                                                     \
                            return launch_blk<NET, float>(a, grid, s);                       \
                    } else if constexpr (y_fits<NET, 256>()) {                               \
                        OV_STAGE_CASE(NET, float, 18)                                        \
                    }                                                                        \
                    if constexpr (y_fits<NET, 128>()) {                                      \
                        OV_STAGE_CASE(NET, float, 20)                                        \
                    }                                                                        \
                    if constexpr (y_fits<NET, 384>()) {                                      \
                        OV_STAGE_CASE(NET, float, 19)                                        \
                    }                                                                        \
                }                                                                            \
                if constexpr (hist_fits_3x128<NET>()) {                                      \
                    OV_STAGE_CASE(NET, float, 21)                                            \
                }                                                                            \
                if constexpr (hist_fits<NET, 256>()) {                                           \
                    OV_STAGE_CASE(NET, float, 9)                                                 \
                }                                                                                \
                if constexpr (hist_fits<NET, 320>()) {                                           \
                    OV_STAGE_CASE(NET, float, 10)                                                \
                }                                                                                \
                if constexpr (hist_fits_max<NET, 384>()) {                                       \
                    OV_STAGE_CASE(NET, float, 12)                                                \
                    OV_STAGE_CASE(NET, float, 17)                                            \
                }                                                                                \
                if constexpr (shm_fits<NET, float, 192>()) {                                     \
                    OV_STAGE_CASE(NET, float, 11)                                                \
                }                                                                                \
                if constexpr (wpc_ok<NET, float, 32>()) {                                    \
                    if (stage == 7)                                                          \
                        return launch_wpc<NET, float, 32>(a, grid, s);                       \
                }                                                                            \
                if constexpr (wpc_ok<NET, float, 16>()) {                                    \
                    if (stage == 13)                                                         \
                        return launch_wpc<NET, float, 16>(a, grid, s);                       \
                }                                                                            \
                if constexpr (wpc_ok<NET, float, 8>()) {                                     \
                    if (stage == 14)                                                         \
                        return launch_wpc<NET, float, 8>(a, grid, s);                        \
                }                                                                            \
                if constexpr (shm_fits<NET, float, 128>()) {                                     \
                    OV_STAGE_CASE(NET, float, 2)                                                 \
                }                                                                                \
                if constexpr (shm_fits<NET, float, 192>()) {                                     \
                    OV_STAGE_CASE(NET, float, 5)                                                 \
                }                                                                                \
                return cudaErrorNotSupported;                                                    \
            }                                                                                    \
            if (G == 32 && lu == 1)                                                              \
                return launch<NET, 32, float, 1>(a, block, grid, s);                             \
        }                                                                                        \
        if (G == 32 && lu == 0)                                                                  \
            return launch<NET, 32, double, 1>(a, block, grid, s);                                \
        return cudaErrorNotSupported;                                                            \
    }                                                                                            \
    }                                                                                            \
    }
