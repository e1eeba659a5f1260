/* The BDF integrator with a block of eight warps integrating 32 cells at a
 * time, for large networks (staging 18).
 *
 * One thread per cell cannot hold a cell of a large network: SYN64's history,
 * factors and vectors are 7 to 9 KB, which stream through local memory, and
 * one trip of a warp's 32 cells is one long chain of instructions.  Here lane
 * l of all eight warps works on the same cell, and the warps share its
 * species: warp w holds the Nordsieck history, correction and previous
 * correction of ND/8 species in registers and does their share of every
 * vector operation (and, without contraction, their rows of the right-hand
 * side and a share of the iteration matrix, BLK_SPLIT below).  The state, the
 * residual, the correction, the weights and the packed factors lie in shared
 * memory, so nothing of a cell is in local or global memory while it runs.
 * The factorisation and the triangular solves, whose statements depend on one
 * another from species to species, run in one warp for all 32 cells; the
 * norms are summed in species order, each by one warp.  What decides a cell's
 * course (time, step, order, phase, counters) is kept by every warp: all
 * compute it from the same sums, so they agree without exchanging it.
 *
 * Every value is the product of the same IEEE operations in the same order
 * as in bdf_kernel.cuh, whose phases (Phase, SsMode) and network code this
 * kernel shares; results equal its results bit for bit.
 *
 * Bound by one warp at a time: the others wait at a barrier (9.9 of the stall
 * cycles per issued instruction over all warps) while one walks through its
 * part of some 200 KB of straight-line network code, at about 16 cycles per
 * instruction in the solve, the right-hand side and the factorisation;
 * instruction fetch is 2.6 of the stall cycles, and no counter shows the
 * working warp alone.  No memory traffic to speak of.  SYN64 against a thread
 * per cell in 256-thread blocks with the state in shared memory, B200: 65,536
 * cells FP32-LU 451 -> 245 ms, FP64 575 -> 515 ms, FP64 with contraction 511 ->
 * 428 ms; 3,001 cells FP32-LU 130 -> 25 ms, FP64 157 -> 38 ms; 64 cells FP64
 * 121 -> 18 ms.
 *
 * Barriers: every warp runs the same trip, and every condition around a
 * barrier is the same in all warps (ballots over state that all warps hold
 * alike, or words read from shared memory after a barrier).  All loops are
 * bounded as in bdf_kernel.cuh. */
#pragma once

namespace ov {
namespace OV_MODE_NS {

constexpr int BLK_WARPS = 8;
/* idle lanes take new cells on every BLK_REFILL-th trip; the Jacobian and
   step-size blocks run on every BLK_PERIOD-th trip (or when no lane can
   progress otherwise), as in bdf_kernel.cuh */
constexpr unsigned BLK_REFILL = 4, BLK_PERIOD = 4;
/* Without contraction every warp evaluates its species' rows of the
   right-hand side and its share of the matrix.  With it the sums must be
   compiled whole, each in one warp: which product of a sum is rounded on its
   own depends on how often the surrounding code uses it, and a divided
   function gave other last bits (4 of SYN64's 64 rows). */
#if defined(OV_FUSED)
constexpr bool BLK_SPLIT = false;
#else
constexpr bool BLK_SPLIT = true;
#endif

/* Without contraction a thread per cell (staging 18's other form) is the faster
   one from two cells per lane on, in blocks of 256: its divisions run for 32
   cells beside seven other warps' work, here in one warp while the others
   wait.  SYN64 FP64 on 148 SMs, thread per cell / block per 32 cells: 3,001
   cells 157 / 38 ms, 37,888 cells 290 / 302, 65,536 cells 526 / 521, 75,776
   cells (the line) 560 / 599, 262,144 cells 1,810 / 2,060.  The one size in
   between where a thread per cell is ahead as well, by 4 %, is that of one cell
   for every lane.  (With contraction 262,144 cells take 1,624 ms here against
   1,910, FP32-LU 944 against 1,530.) */
constexpr int BLK_SPLIT_THREADS = 256;
constexpr int64_t blk_split_cells(int sms) { return (int64_t)2 * sms * BLK_SPLIT_THREADS; }

template <class Net, class LUT>
struct BlkLayout {
    static constexpr int ND = Net::ND;
    static constexpr int NS = (ND + BLK_WARPS - 1) / BLK_WARPS; /* species per warp */
    static constexpr int ROW = ND | 1; /* odd: a warp's accesses to one species spread over the banks */
    static constexpr size_t lu_bytes = sizeof(LUT) * Net::NNZ * 32;
    static constexpr size_t lu_pad = (lu_bytes + 15) / 16 * 16;
    static constexpr size_t row_bytes = sizeof(double) * 32 * ROW;
    static constexpr size_t smem_bytes = lu_pad + 5 * row_bytes; /* rows Y, R, D, E, W */
};

/* networks the kernel is compiled for: constant coefficients, a symbolic
   Jacobian, every species in the solver state, more species than a thread
   can hold, and the arrays of 32 cells within a block's shared memory */
template <class Net, class LUT>
constexpr bool blk_ok()
{
    return Net::ND > 32 && Net::ND <= 64 && Net::NF == 0 && Net::NREA == 0 && Net::LU_METHOD == 1 && !Net::HC_FD &&
           !Net::HEATCOOL && BlkLayout<Net, LUT>::smem_bytes <= 226 * 1024;
}

struct BlkShared {
    double sum[3][32];
    unsigned long long base;
    int stop;
    unsigned pneg[BLK_WARPS], neg[BLK_WARPS], nan[BLK_WARPS];
};

__device__ __forceinline__ void blk_sync()
{
    __syncwarp();
    __syncthreads();
}

/* rows W*NS.. of the right-hand side: the other rows' statements are unused
   and fall away */
template <class Net, int W, int NS>
__device__ __forceinline__ void blk_rhs_rows(const double* y, double* f)
{
    double all[Net::NEQ];
    Net::rhs(y, nullptr, all);
#pragma unroll
    for (int i = 0; i < NS; ++i)
        if (W * NS + i < Net::ND)
            f[i] = all[W * NS + i];
        else
            f[i] = 0.0;
}

template <class Net, int NS>
__device__ __forceinline__ void blk_rhs(int w, const double* y, double* f)
{
    switch (w) {
    case 0: blk_rhs_rows<Net, 0, NS>(y, f); break;
    case 1: blk_rhs_rows<Net, 1, NS>(y, f); break;
    case 2: blk_rhs_rows<Net, 2, NS>(y, f); break;
    case 3: blk_rhs_rows<Net, 3, NS>(y, f); break;
    case 4: blk_rhs_rows<Net, 4, NS>(y, f); break;
    case 5: blk_rhs_rows<Net, 5, NS>(y, f); break;
    case 6: blk_rhs_rows<Net, 6, NS>(y, f); break;
    default: blk_rhs_rows<Net, 7, NS>(y, f); break;
    }
}

/* packed matrix entries [LO, HI) of a lane's column in shared memory; writes
   to the others go to a word nobody reads, so their statements fall away */
template <class T, int LO, int HI>
struct LanePart {
    T* base;
    T* none;
    __device__ __forceinline__ T& operator[](int i) const { return i >= LO && i < HI ? base[i * 32] : *none; }
};

template <class Net, int W>
__device__ __forceinline__ void blk_jac_part(const double* y, double beta, double h, double* lu)
{
    constexpr int LO = Net::NNZ * W / BLK_WARPS, HI = Net::NNZ * (W + 1) / BLK_WARPS;
    double none;
    Net::template jac<double>(y, nullptr, beta, h, LanePart<double, LO, HI>{lu, &none});
}

template <class Net>
__device__ __forceinline__ void blk_jac(int w, const double* y, double beta, double h, double* lu)
{
    switch (w) {
    case 0: blk_jac_part<Net, 0>(y, beta, h, lu); break;
    case 1: blk_jac_part<Net, 1>(y, beta, h, lu); break;
    case 2: blk_jac_part<Net, 2>(y, beta, h, lu); break;
    case 3: blk_jac_part<Net, 3>(y, beta, h, lu); break;
    case 4: blk_jac_part<Net, 4>(y, beta, h, lu); break;
    case 5: blk_jac_part<Net, 5>(y, beta, h, lu); break;
    case 6: blk_jac_part<Net, 6>(y, beta, h, lu); break;
    default: blk_jac_part<Net, 7>(y, beta, h, lu); break;
    }
}

/* the packed factors of a lane's cell in shared memory, for a factorisation or
   a solve without scheduling fences: the band of entries in use stays in
   registers (SYN64, 65,536 cells, FP64: 497 against 515 ms with fences) */
template <class T>
struct BlkCol {
    T* base;
    __device__ __forceinline__ T& operator[](int i) const { return base[i * 32]; }
};

}  // namespace OV_MODE_NS
}  // namespace ov

template <class T>
struct ov_lu_fenced<ov::OV_MODE_NS::BlkCol<T>> {
    static constexpr bool value = false;
};

namespace ov {
namespace OV_MODE_NS {

/* sum of e_j^2 w_j in species order (the norms' order, src/odevec.F90:669-702) */
template <int ND>
__device__ __forceinline__ double blk_sum_sq(const double* e, const double* w)
{
    double s = 0.0;
#pragma unroll 16
    for (int j = 0; j < ND; ++j)
        s = s + e[j] * e[j] * w[j];
    return s;
}

template <class Net, class LUT>
__device__ __forceinline__ void blk_run(const LaunchArgs& A)
{
    using L = BlkLayout<Net, LUT>;
    constexpr int ND = L::ND, NS = L::NS, ROW = L::ROW;
    constexpr bool SCALED = sizeof(LUT) == 4;
    constexpr bool EVEN = ND % BLK_WARPS == 0; /* every warp has NS species */
    if (A.run_if && *A.run_if == 0)
        return;
    extern __shared__ __align__(16) unsigned char ov_smem[];
    __shared__ BlkShared sm;
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const int j0 = w * NS;
    LUT* const lu = reinterpret_cast<LUT*>(ov_smem) + lane;
    double* const rows = reinterpret_cast<double*>(ov_smem + L::lu_pad) + (size_t)lane * ROW;
    double* const Y = rows;                /* state */
    double* const R = rows + 32 * ROW;     /* residual; scale of the Jacobian */
    double* const D = rows + 2 * 32 * ROW; /* correction; inverse scale */
    double* const E = rows + 3 * 32 * ROW; /* accumulated correction, for the sums */
    double* const Wt = rows + 4 * 32 * ROW; /* error weights */
    auto own = [&](int i) { return EVEN || j0 + i < ND; };
    auto div_n = [](double x) {
        if constexpr ((Net::NEQ & (Net::NEQ - 1)) == 0)
            return x * (1.0 / Net::NEQ);
        else
            return x / Net::NEQ;
    };

    const int64_t ncells = A.ncells, stride = A.stride;
    double yns[MAXQ + 1][NS], en[NS], eno[NS];
    short sce[SCALED ? NS : 1];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        en[i] = eno[i] = 0.0;
#pragma unroll
        for (int k = 0; k <= MAXQ; ++k)
            yns[k][i] = 0.0;
        if constexpr (SCALED)
            sce[i] = 0;
    }
    double t = 0, h = 0, told = 0, tstop = 0, crate = 0, jchg = 0, cerr = 0, tint = 0;
    int q = 1, swu = 0, lju = 0, fet = 0, fc = 0, it = 0, ss_mode = 0;
    bool ujac = false, nuo = false, first = false, msk = true, write_y = false;
    int status = OV_OK, attempts = 0, steps = 0, ltef = 0, convf = 0, newt = 0, jacs = 0, ppass = 0;
    int ph = A.lanes > 0 && lane >= A.lanes ? PH_EXHAUSTED : PH_IDLE;
    int64_t cell = -1;
    __syncthreads(); /* a block may come from another job */

    /* the warp's share of the per-cell steps of bdf_kernel.cuh */
    auto weights = [&]() {
        unsigned odd = 0;
        double v[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const double x = own(i) ? A.rtol * fabs(Y[j0 + i]) + A.atol : 1.0;
            odd |= rcp_odd(x);
            v[i] = rcp_normal(x);
        }
        if (odd) {
#pragma unroll
            for (int i = 0; i < NS; ++i)
                v[i] = __drcp_rn(own(i) ? A.rtol * fabs(Y[j0 + i]) + A.atol : 1.0);
        }
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (own(i))
                Wt[j0 + i] = v[i] * v[i];
    };
    auto reset = [&]() { /* ResetSystem (src/odevec.F90:526-544) */
        ppass += q * (q + 1) / 2;
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
            for (int k = 0; k < MAXQ; ++k)
#pragma unroll
                for (int jj = MAXQ; jj >= 1; --jj)
                    if (k <= q - 1 && jj <= q && jj >= k + 1)
                        yns[jj - 1][i] = yns[jj - 1][i] - yns[jj][i];
    };
    auto set_step = [&](double dt_scale) { /* SetStepSize (src/odevec.F90:720-743) */
        double dtt = 1.0;
#pragma unroll
        for (int k = 1; k <= MAXQ; ++k) {
            dtt = dt_scale * dtt;
            if (k <= q) {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    yns[k][i] = yns[k][i] * dtt;
            }
        }
        h = h * dt_scale;
        jchg = jchg * dt_scale;
    };
    auto interpolate = [&]() { /* InterpolateSolution (src/odevec.F90:998-1030) */
        const double rel_t = (tstop - t) / h;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            double acc = yns[MAXQ][i];
#pragma unroll
            for (int k = MAXQ - 1; k >= 0; --k) {
                const double next = yns[k][i] + rel_t * acc;
                acc = k < q ? next : yns[k][i];
            }
            if (own(i))
                Y[j0 + i] = acc;
        }
    };
    auto finish_step = [&]() { /* src/odevec.F90:452-464, loop test :207 */
        fet = 0;
        steps++;
        if (lju >= 20)
            ujac = true;
        else if (fabs(jchg - (double)1.0f) > (double)0.3f)
            ujac = true;
#pragma unroll
        for (int i = 0; i < NS; ++i)
            eno[i] = en[i];
        if (t < tstop) {
            told = t;
            ph = PH_PRED;
        } else {
            write_y = true;
            interpolate();
            tint = t;
            t = tstop;
            ph = PH_DONE;
        }
    };
    auto restart_state = [&]() {
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if (own(i))
                Y[j0 + i] = yns[0][i];
    };

    unsigned trip = 0;
    for (;;) {
        /* ---- 1. idle lanes take new cells ---------------------------- */
        {
            const bool refill = trip % BLK_REFILL == 0u;
            const bool ask = refill && trip > 0u && A.yield;
            unsigned need = refill ? __ballot_sync(FULL, ph == PH_IDLE) : 0u;
            ++trip;
            if (need) {
                if (threadIdx.x == 0) {
                    const int stop = ask ? *(volatile const int32_t*)A.yield : 0;
                    sm.stop = stop;
                    if (!stop)
                        sm.base = atomicAdd(A.queue, (unsigned long long)__popc(need));
                }
                blk_sync();
                if (sm.stop) {
                    if (ph == PH_IDLE)
                        ph = PH_EXHAUSTED;
                } else if (ph == PH_IDLE) {
                    const int64_t k = (int64_t)(sm.base + __popc(need & ((1u << lane) - 1u)));
                    if (k < ncells) {
                        cell = A.order ? (int64_t)A.order[k] : k;
                        ph = PH_START;
                    } else {
                        ph = PH_EXHAUSTED;
                    }
                }
            }
            if (__all_sync(FULL, ph == PH_EXHAUSTED))
                break;
        }

        /* ---- load + SolveODE set-up (src/odevec.F90:169-198) --------- */
        if (ph == PH_START) {
            t = A.t[cell];
            h = A.dt[cell];
#pragma unroll
            for (int i = 0; i < NS; ++i)
                if (own(i)) {
                    const double v = A.y[(int64_t)(j0 + i) * stride + cell];
                    Y[j0 + i] = v;
                    if (A.save_y)
                        A.save_y[(int64_t)(j0 + i) * ncells + cell] = v;
                }
            if (A.save_y && w == 0) {
                A.save_t[cell] = t;
                A.save_dt[cell] = h;
            }
            tstop = A.t_stop[cell];
            msk = A.mask ? (A.mask[cell] != 0) : true;
            status = OV_OK;
            attempts = steps = ltef = convf = newt = jacs = ppass = 0;
            first = true;
            q = 1;
            swu = 0;
            crate = 0.7;
            jchg = 0.0;
            nuo = false;
            fet = 0;
            fc = 0;
            ujac = true;
            lju = 0;
            cerr = 0.0;
            it = 0;
            ss_mode = 0;
            write_y = false;
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                eno[i] = 0.0;
#pragma unroll
                for (int k = 0; k <= MAXQ; ++k)
                    yns[k][i] = 0.0;
            }
            weights();
            if (!msk) {
                t = tstop; /* src/odevec.F90:187-191 */
                ph = PH_DONE;
            } else if (A.resume == 1) {
                const double* ws = A.ws;
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i)) {
#pragma unroll
                        for (int k = 0; k <= MAXQ; ++k)
                            yns[k][i] = ws[((int64_t)k * ND + j0 + i) * stride + cell];
                        eno[i] = ws[((int64_t)(MAXQ + 1) * ND + j0 + i) * stride + cell];
                        Wt[j0 + i] = ws[((int64_t)(MAXQ + 2) * ND + j0 + i) * stride + cell];
                        Y[j0 + i] = yns[0][i];
                    }
                const double* s = ws + (int64_t)(MAXQ + 3) * ND * stride + cell;
                t = s[0];
                h = s[stride];
                crate = s[2 * stride];
                jchg = s[3 * stride];
                q = (int)s[4 * stride];
                swu = (int)s[5 * stride];
                lju = (int)s[6 * stride];
                fet = (int)s[7 * stride];
                fc = (int)s[8 * stride];
                nuo = s[10 * stride] != 0.0;
                first = s[11 * stride] != 0.0;
                ujac = true;
                if (t < tstop) {
                    told = t;
                    ph = PH_PRED;
                } else {
                    write_y = true;
                    interpolate();
                    tint = t;
                    t = tstop;
                    ph = PH_DONE;
                }
            } else {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i)) {
                        if (A.resume == 2)
                            eno[i] = A.ws[((int64_t)(MAXQ + 1) * ND + j0 + i) * stride + cell];
                        yns[0][i] = Y[j0 + i];
                    }
            }
        }

        /* ---- 2. predictor attempt (src/odevec.F90:259-299) ----------- */
        {
            bool tried = false, neg = false;
            if (ph == PH_PRED) {
                if (++attempts > A.max_attempts) {
                    status = OV_ERR_MAX_STEPS;
                    ph = PH_DONE;
                } else {
                    tried = true;
                    t = t + h;
                    ppass += q * (q + 1) / 2;
#pragma unroll
                    for (int i = 0; i < NS; ++i) {
#pragma unroll
                        for (int l = 0; l < MAXQ; ++l)
#pragma unroll
                            for (int k = MAXQ; k >= 1; --k)
                                if (l <= q - 1 && k <= q && k >= l + 1)
                                    yns[k - 1][i] = yns[k][i] + yns[k - 1][i];
                        en[i] = 0.0;
                        neg |= own(i) && yns[0][i] < 0.0;
                    }
                }
            }
            if (A.check_neg) {
                const unsigned b = __ballot_sync(FULL, tried && neg);
                if (lane == 0)
                    sm.pneg[w] = b;
                blk_sync();
                unsigned any = 0;
#pragma unroll
                for (int k = 0; k < BLK_WARPS; ++k)
                    any |= sm.pneg[k];
                neg = (any >> lane) & 1u;
            } else {
                neg = false;
            }
            if (tried) {
                if (neg) {
                    t = told;
                    reset();
                    set_step(0.25);
                    if (h <= A.dt_min) {
                        status = OV_ERR_DTMIN_PREDICTOR;
                        ph = PH_DONE;
                    }
                } else {
                    restart_state();
                    it = 0;
                    ph = ujac ? PH_JACWAIT : PH_NEWTON;
                }
            }
        }
        blk_sync(); /* the state is complete */

        /* ---- 3. Jacobian + LU for the waiting lanes (:301-315) ------- */
        bool jac = false;
        {
            const int waiting = warp_count(ph == PH_JACWAIT);
            const int moving = warp_count(ph == PH_NEWTON || ph == PH_START || ph == PH_RESTART);
            const bool run = waiting > 0 && (trip % BLK_PERIOD == 1u % BLK_PERIOD || moving == 0);
            jac = run && ph == PH_JACWAIT;
            if (SCALED && run) {
                if (jac) {
                    /* powers of two close to the error weights */
#pragma unroll
                    for (int i = 0; i < NS; ++i)
                        if (own(i)) {
                            int e = (int)((ov_d2bits(Wt[j0 + i]) >> 52) & 0x7ff) - 1023;
                            int hexp = e >= 0 ? e / 2 : -((-e + 1) / 2);
                            hexp = hexp > 480 ? 480 : (hexp < -480 ? -480 : hexp);
                            sce[SCALED ? i : 0] = (short)hexp;
                            R[j0 + i] = ov_pow2i(hexp);
                            D[j0 + i] = ov_pow2i(-hexp);
                        }
                }
                blk_sync();
            }
            if constexpr (BLK_SPLIT) {
                /* every warp its share of the matrix */
                if (run) {
                    if (jac)
                        blk_jac<Net>(w, Y, lcoef(q, 0), h, lu);
                    blk_sync();
                }
            } else if (jac && w == 1) {
                /* one warp, while another evaluates the right-hand side */
                if constexpr (SCALED)
                    Net::template jac_scaled<LUT>(Y, nullptr, lcoef(q, 0), h, LaneCol<LUT, 32>{lu}, R, D);
                else
                    Net::template jac<LUT>(Y, nullptr, lcoef(q, 0), h, LaneCol<LUT, 32>{lu});
            }
            if (jac && w == 1)
                Net::template lu_factor<LUT>(BlkCol<LUT>{lu});
            if (jac) {
                jacs++;
                ujac = false;
                lju = 0;
                crate = 0.7;
                jchg = 1.0;
                ph = PH_NEWTON;
            }
        }

        /* ---- 4. right-hand side, residual ---------------------------- */
        const bool evaluating = ph == PH_START || ph == PH_NEWTON || ph == PH_RESTART;
        if constexpr (!BLK_SPLIT) {
            if (evaluating && w == 0)
                Net::rhs(Y, nullptr, E);
            blk_sync();
        }
        if (evaluating) {
            double f[NS];
            if constexpr (BLK_SPLIT) {
                blk_rhs<Net, NS>(w, Y, f);
            } else {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    f[i] = own(i) ? E[j0 + i] : 0.0;
            }
            if (ph == PH_NEWTON) {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i)) {
                        double res = h * f[i] - (yns[1][i] + en[i]);
                        if constexpr (SCALED)
                            res = res * ov_pow2i(sce[i]);
                        R[j0 + i] = res;
                    }
            } else {
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    yns[1][i] = h * f[i];
                    if (own(i))
                        R[j0 + i] = f[i];
                }
            }
        }
        const bool starting = ph == PH_START, solving = ph == PH_NEWTON;
        if (ph == PH_RESTART) { /* src/odevec.F90:417-421 */
            ujac = true;
            ss_mode = SS_RESTART;
            ph = PH_SSWAIT;
        }
        blk_sync(); /* the residual is complete */

        /* ---- 5. solve; initial step size ----------------------------- */
        if (solving && w == 0)
            Net::template lu_solve<LUT>(BlkCol<LUT>{lu}, R, D, nullptr, nullptr);
        if (starting && w == 1) {
            /* CalcInitialStepSize (src/odevec.F90:216-238) */
            const double tol = A.rtol;
            double s = 0.0;
#pragma unroll 8
            for (int j = 0; j < ND; ++j)
                s = s + R[j] * R[j] * (Wt[j] * tol * tol);
            sm.sum[2][lane] = s;
        }
        blk_sync(); /* the correction is complete */
        if (starting) {
            const double mx = max_operand(sm.sum[2][lane]);
            const double W0 = fabs(t) > fabs(tstop) ? fabs(t) : fabs(tstop);
            const double d = sqrt(A.rtol / (ov_pow(W0, -2.0) + div_n(mx)));
            const double span = fabs(tstop - t);
            h = d < span ? d : span;
            if (t < tstop) {
                told = t;
                ph = PH_PRED;
            } else {
                write_y = true;
                interpolate();
                tint = t;
                t = tstop;
                ph = PH_DONE;
            }
        }
        {
            bool neg = false, nan = false;
            if (solving) {
                newt++;
                const double l0 = lcoef(q, 0);
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i)) {
                        double den = D[j0 + i];
                        if constexpr (SCALED) {
                            den = den * ov_pow2i(-sce[i]);
                            D[j0 + i] = den;
                        }
                        en[i] = en[i] + den;
                        const double y = yns[0][i] + l0 * en[i];
                        Y[j0 + i] = y;
                        E[j0 + i] = en[i];
                        neg |= y < 0.0;
                        const double wt = Wt[j0 + i];
                        nan |= (den != den) | (wt != wt);
                    }
            }
            const unsigned bn = __ballot_sync(FULL, nan), bg = __ballot_sync(FULL, neg);
            if (lane == 0) {
                sm.nan[w] = bn;
                sm.neg[w] = bg;
            }
        }
        blk_sync(); /* the new state and the correction are complete */

        /* ---- 6. norms, convergence and error tests ------------------- */
        if (solving) {
            if (w == 0)
                sm.sum[0][lane] = blk_sum_sq<ND>(D, Wt);
            else if (w == 1)
                sm.sum[1][lane] = blk_sum_sq<ND>(E, Wt);
        }
        blk_sync(); /* the sums are complete */
        if (solving) {
            const double s_lane = sm.sum[0][lane];
            unsigned any_nan = 0, any_neg = 0;
#pragma unroll
            for (int k = 0; k < BLK_WARPS; ++k) {
                any_nan |= sm.nan[k];
                any_neg |= sm.neg[k];
            }
            /* CheckConvergence (src/odevec.F90:622-665) */
            bool failed = false, converged = false;
            const double err = max_operand(sqrt(div_n(s_lane)));
            double rate_tmp = 0.0;
            if (it != 0) {
                rate_tmp = err / cerr;
                crate = fmax(0.2 * crate, rate_tmp);
            }
            const double r15 = 1.5 * crate;
            const double crit = err * (1.0 < r15 ? 1.0 : r15);
            if (s_lane != s_lane && ((any_nan >> lane) & 1u)) {
                failed = true;
            } else if (crit < conv_divisor(q)) {
                converged = true;
            } else if (it >= 2 && crate > 2.0 * rate_tmp) {
                failed = true;
            } else if (it == 3) {
                failed = true;
            } else {
                cerr = err;
                it = it + 1;
            }
            if (A.check_neg && ((any_neg >> lane) & 1u)) {
                failed = true;
                converged = false;
            }
            if (failed && !converged) {
                /* src/odevec.F90:375-393 */
                t = told;
                fc++;
                convf++;
                if (fc > 10) {
                    status = OV_ERR_CONV_FAILURES;
                    ph = PH_DONE;
                } else {
                    it = 0;
                    reset();
                    set_step(0.25);
                    if (h < A.dt_min) {
                        status = OV_ERR_DTMIN_CONV;
                        ph = PH_DONE;
                    } else {
                        ujac = true;
                        ph = PH_PRED;
                    }
                }
            } else if (converged) {
                fc = 0;
                /* local truncation error test (src/odevec.F90:400-455) */
                const bool lte = max_operand(div_n(sm.sum[1][lane])) >= c_lte[q];
                weights();
                if (lte) {
                    ltef++;
                    t = told;
                    if (fet >= 3) {
                        if (A.fix_restart)
                            reset();
                        q = 1;
                        restart_state();
                        ph = PH_RESTART;
                    } else {
                        reset();
                        ujac = true;
                        swu = 0;
                        nuo = true;
                        ss_mode = SS_REJECT;
                        ph = PH_SSWAIT;
                    }
                } else {
                    swu++;
                    lju++;
                    /* UpdateNordsieck (src/odevec.F90:747-765) */
#pragma unroll
                    for (int k = 0; k <= MAXQ; ++k)
                        if (k <= q) {
                            const double c = lcoef(q, k);
#pragma unroll
                            for (int i = 0; i < NS; ++i)
                                yns[k][i] = yns[k][i] + en[i] * c;
                        }
                    if (swu == q + 1) {
                        ss_mode = SS_ACCEPT;
                        ph = PH_SSWAIT;
                    } else {
                        finish_step();
                    }
                }
            }
        }

        /* ---- 7. step-size / order selection for the waiting lanes --- */
        {
            const int waiting = warp_count(ph == PH_SSWAIT);
            const int moving = warp_count(ph == PH_PRED || ph == PH_NEWTON || ph == PH_RESTART);
            const bool run = waiting > 0 && (trip % BLK_PERIOD == 0u || moving == 0);
            if (run) {
                const bool mine = ph == PH_SSWAIT;
                if (mine) {
#pragma unroll
                    for (int i = 0; i < NS; ++i)
                        if (own(i)) {
                            double v = yns[1][i];
#pragma unroll
                            for (int k = 2; k <= MAXQ; ++k)
                                v = k == q ? yns[k][i] : v;
                            R[j0 + i] = v;
                            D[j0 + i] = en[i] - eno[i];
                            E[j0 + i] = en[i];
                        }
                }
                blk_sync();
                if (mine && w < 3)
                    sm.sum[w][lane] = blk_sum_sq<ND>(w == 0 ? R : (w == 1 ? E : D), Wt);
                blk_sync();
                if (mine) {
                    const int order = q;
                    int loc;
                    bool big;
                    double s = step_choice(order, order != 1, !(order == MAXQ || nuo),
                                           max_operand(div_n(sm.sum[0][lane])), max_operand(div_n(sm.sum[1][lane])),
                                           max_operand(div_n(sm.sum[2][lane])), loc, big);
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
                                for (int k = 2; k <= MAXQ; ++k)
                                    if (k == order + 1) {
#pragma unroll
                                        for (int i = 0; i < NS; ++i)
                                            yns[k][i] = c * en[i] / (order + 1.0);
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
                    if (status) {
                        ph = PH_DONE;
                    } else {
                        set_step(s);
                        if (ss_mode == SS_ACCEPT) {
                            finish_step();
                        } else {
                            fet++; /* src/odevec.F90:434-439 */
                            ph = PH_PRED;
                        }
                    }
                }
            }
        }

        /* ---- 8. store finished cells -------------------------------- */
        if (ph == PH_DONE) {
            const bool ok = status == OV_OK;
            if (A.ws && ok && write_y) {
                double* ws = A.ws;
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i)) {
#pragma unroll
                        for (int k = 0; k <= MAXQ; ++k)
                            ws[((int64_t)k * ND + j0 + i) * stride + cell] = yns[k][i];
                        ws[((int64_t)(MAXQ + 1) * ND + j0 + i) * stride + cell] = eno[i];
                        ws[((int64_t)(MAXQ + 2) * ND + j0 + i) * stride + cell] = Wt[j0 + i];
                    }
                if (w == 0) {
                    double* s = ws + (int64_t)(MAXQ + 3) * ND * stride + cell;
                    const double sc[12] = {tint, h, crate, jchg, (double)q, (double)swu, (double)lju, (double)fet,
                                           (double)fc, ujac ? 1.0 : 0.0, nuo ? 1.0 : 0.0, first ? 1.0 : 0.0};
#pragma unroll
                    for (int i = 0; i < 12; ++i)
                        s[i * stride] = sc[i];
                }
            }
            if ((!ok || write_y) && msk) {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (own(i))
                        A.y[(int64_t)(j0 + i) * stride + cell] = Y[j0 + i];
            }
            if (w == 0) {
                A.t[cell] = t;
                A.dt[cell] = h;
                if (A.status)
                    A.status[cell] = status;
                if (A.stats) {
                    int32_t* s = A.stats + cell * OV_NSTATS;
                    s[0] = steps;
                    s[1] = attempts;
                    s[2] = ltef;
                    s[3] = convf;
                    s[4] = newt;
                    s[5] = jacs;
                    s[6] = q;
                    s[7] = ppass;
                }
            }
            ph = PH_IDLE;
        }
    }
}

template <class Net, class LUT>
__global__ void __launch_bounds__(32 * BLK_WARPS, 1) blk_kernel(const __grid_constant__ LaunchArgs A)
{
    blk_run<Net, LUT>(A);
}

/* One block per SM, 32 cells each; fewer cells per block where that fills
   all SMs (a trip takes the same time for one cell as for 32, but its lanes
   wait for one another at the Jacobian and step-size blocks). */
template <class Net, class LUT>
cudaError_t launch_blk(const LaunchArgs& a, int grid, cudaStream_t stream)
{
    auto kern = blk_kernel<Net, LUT>;
    constexpr size_t smem = BlkLayout<Net, LUT>::smem_bytes;
    int sms = 0;
    cudaError_t err = device_sms(&sms);
    if (err == cudaSuccess)
        err = allow_smem((const void*)kern, smem);
    if (err != cudaSuccess)
        return err;
    LaunchArgs b = a;
    if (grid <= 0) {
        int64_t lanes = (a.ncells + sms - 1) / sms;
        b.lanes = (int32_t)(lanes < 32 ? lanes : 32);
        const int64_t want = (a.ncells + b.lanes - 1) / b.lanes;
        grid = (int)(want < sms ? want : sms);
    }
    kern<<<grid, 32 * BLK_WARPS, smem, stream>>>(b);
    return cudaGetLastError();
}

}  // namespace OV_MODE_NS
}  // namespace ov
