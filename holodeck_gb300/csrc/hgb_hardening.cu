// Binary hardening on the GPU:
//  * hgb_find_2pwl_hardening_norm: Brent root of the two-power-law lifetime per (mtot, mrat) cell
//    (holodeck/sams/sam_cyutils.pyx:289-398).  k_hardening_norm_sub: two or four cells a warp, the nodes of a
//    total mass shared by a block; k_hardening_norm, a warp per cell, beyond its 320 steps.
//  * hgb_dbn_2pwl: differential binary number for Fixed_Time_2PL_SAM (sam_cyutils.pyx:510-781) in two phases.
//    The first records, per starting redshift and target frequency, the interpolated time of the separation
//    step that brackets the target: k_dbn_2pwl_walk for ascending targets (several mrat cells of one mtot a
//    block; steps found in FP32, brackets evaluated in FP64), k_dbn_2pwl for targets in any order, or tables
//    beyond the first's limits.  k_dbn_2pwl_eval then evaluates redshift, distance, residence time and number
//    of every bracketed (redz, frequency) element, the model's (half-)integer exponents as products and
//    roots instead of pow().  The age -> redshift / distance interpolations use per-interval slopes computed
//    once per block (a multiply instead of a divide per lookup; an ulp from the reference's divide).
//  * hgb_dbn_gw: differential binary number for Hard_GW (sam_cyutils.pyx:788-899); one block per
//    run of up to 256 (mtot, mrat, redz) points.
// FP64 throughout (the hardening integral and the lookback-time -> redshift inversion are the
// FP64 islands of the path).  Built with -fmad=false: k_hardening_norm, k_dbn_2pwl and the walk's nodes and
// running times keep the reference loops' order and rounding, to the last-ulp behaviour of pow/log10.  The
// other kernels regroup: explicit multiply-adds, fast_rcp / fast_rsqrt for quotients and roots, shared powers.
#include <math.h>

#include <algorithm>

#include "hgb_common.cuh"

namespace {

using hgb::CyConst;

constexpr double NORM_LOG10_LO = -20.0;
constexpr double NORM_LOG10_HI = +20.0;
constexpr double BRENT_XTOL = 1e-3;
constexpr double BRENT_RTOL = 1e-5;
constexpr int BRENT_MAXITER = 100;

// ------------------------------------------------------------------------------------------------
// hardening normalisation
// ------------------------------------------------------------------------------------------------

struct PowPlan {
    int kind;   // 0: pow(), 1: integer, 2: half-integer
    int n;      // |y| rounded down
    int neg;    // y < 0
};

struct NormArgs {
    double target_time, sepa_init_log10, rchar, gi, go;
    int nsteps;
    PowPlan p_outer, p_inner;   // exponents -go + gi and gi - 1 of the hardening rate
};

// Lifetime minus target for one cell, evaluated by the whole warp (sam_cyutils.pyx:360-398).
// sepa/aa/bb/gw hold, per separation node, the norm-independent pieces of the hardening rate;
// the trapezoid terms are formed in parallel and summed in step order by lane 0 so the sum
// rounds like the reference loop.
__device__ double warp_lifetime(double norm_log10, const NormArgs &a, const double *sepa, const double *aa,
                                const double *bb, const double *gw, double *dt, int lane) {
    double norm = pow(10.0, norm_log10);
    for (int s = lane; s < a.nsteps; s += 32) {
        double dl = -norm * aa[s] / bb[s];
        dl += gw[s];
        double dr = -norm * aa[s + 1] / bb[s + 1];
        dr += gw[s + 1];
        dt[s] = 2.0 * (sepa[s + 1] - sepa[s]) / (dl + dr);
    }
    __syncwarp();
    double time = 0.0;
    if (lane == 0) {
        for (int s = 0; s < a.nsteps; s++) time += dt[s];
    }
    time = __shfl_sync(0xffffffffu, time, 0);
    __syncwarp();
    return time - a.target_time;
}

// Brent's method (Brent 1973, "Algorithms for Minimization without Derivatives", ch. 4) with the
// tolerance delta = (xtol + rtol |b|) / 2; returns 0 when the interval does not bracket a root
// and the last iterate when the iteration budget runs out.  All lanes run it in lock step.
__device__ double warp_brent(const NormArgs &a, const double *sepa, const double *aa, const double *bb,
                             const double *gw, double *dt, int lane, int *n_iter_out) {
    double xa = NORM_LOG10_LO, xb = NORM_LOG10_HI;
    double fa = warp_lifetime(xa, a, sepa, aa, bb, gw, dt, lane);
    double fb = warp_lifetime(xb, a, sepa, aa, bb, gw, dt, lane);
    *n_iter_out = 0;
    if (fa * fb > 0.0) return 0.0;
    if (fa == 0.0) return xa;
    if (fb == 0.0) return xb;
    double xc = xa, fc = fa;
    double d = xb - xa, e = d;
    for (int it = 0; it < BRENT_MAXITER; it++) {
        *n_iter_out = it + 1;
        if (fb * fc > 0.0) {
            xc = xa;
            fc = fa;
            d = xb - xa;
            e = d;
        }
        if (fabs(fc) < fabs(fb)) {
            xa = xb; xb = xc; xc = xa;
            fa = fb; fb = fc; fc = fa;
        }
        double tol = 0.5 * (BRENT_XTOL + BRENT_RTOL * fabs(xb));
        double m = 0.5 * (xc - xb);
        if (fb == 0.0 || fabs(m) < tol) return xb;
        if (fabs(e) > tol && fabs(fb) < fabs(fa)) {
            double s;
            if (xa == xc) {
                s = -fb * (xb - xa) / (fb - fa);                               // secant
            } else {
                double da = (fa - fb) / (xa - xb);
                double dc = (fc - fb) / (xc - xb);
                s = -fb * (fc * dc - fa * da) / (dc * da * (fc - fa));         // inverse quadratic
            }
            if (2.0 * fabs(s) < fmin(fabs(e), 3.0 * fabs(m) - tol)) {
                e = d;
                d = s;
            } else {
                d = m;
                e = m;
            }
        } else {
            d = m;
            e = m;
        }
        xa = xb;
        fa = fb;
        xb = xb + ((fabs(d) > tol) ? d : ((m > 0.0) ? tol : -tol));
        fb = warp_lifetime(xb, a, sepa, aa, bb, gw, dt, lane);
    }
    *n_iter_out = BRENT_MAXITER + 1;
    return xb;
}

__global__ void k_hardening_norm(CyConst cc, NormArgs a, const double *__restrict__ mtot,
                                 const double *__restrict__ mrat, int n, double *__restrict__ norm_log10,
                                 double *__restrict__ norm, int *d_status) {
    extern __shared__ double smem[];
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int nwarps = blockDim.x >> 5;
    int cell = blockIdx.x * nwarps + warp;
    if (cell >= n) return;   // whole warp exits together
    int S = a.nsteps;
    double *sepa = smem + (size_t)warp * 5 * (S + 1);
    double *aa = sepa + (S + 1);
    double *bb = aa + (S + 1);
    double *gw = bb + (S + 1);
    double *dt = gw + (S + 1);
    double mt = mtot[cell], mr = mrat[cell];

    // separation nodes: log10 separation stepped down by repeated subtraction (sam_cyutils.pyx:367-383)
    double risco_log10 = log10(3.0 * HGB_CY_SCHW * mt);
    double dx = (a.sepa_init_log10 - risco_log10) / S;
    if (lane == 0) {
        double sl = a.sepa_init_log10;
        sepa[0] = sl;
        for (int s = 1; s <= S; s++) {
            sl -= dx;
            sepa[s] = sl;
        }
    }
    __syncwarp();
    for (int s = lane; s <= S; s += 32) {
        double sp = pow(10.0, sepa[s]);
        double xx = sp / a.rchar;
        aa[s] = pow(1.0 + xx, -a.go + a.gi);
        bb[s] = pow(xx, a.gi - 1.0);
        gw[s] = hgb::hard_gw(cc.c_dadt, mt, mr, sp);
        sepa[s] = sp;
    }
    __syncwarp();
    int nit;
    double root = warp_brent(a, sepa, aa, bb, gw, dt, lane, &nit);
    if (lane == 0) {
        norm_log10[cell] = root;
        if (norm) norm[cell] = pow(10.0, root);
        if (nit > BRENT_MAXITER) hgb::flag(d_status, HGB_STATUS_ITERATION_LIMIT);
    }
}

// ------------------------------------------------------------------------------------------------
// differential binary number, Fixed_Time_2PL_SAM
// ------------------------------------------------------------------------------------------------

// x^y for an exponent fixed per call.  Integer and half-integer exponents up to |y| = 8.5 (the
// hardening model's defaults give -3.5 and -2) are evaluated as products and one square root,
// within a few ulp of pow(); any other exponent goes to pow().
PowPlan pow_plan(double y) {
    PowPlan p{0, 0, y < 0.0};
    const double ay = fabs(y), twice = 2.0 * ay;
    if (ay <= 8.5 && twice == floor(twice)) {
        p.n = (int)floor(ay);
        p.kind = (ay == floor(ay)) ? 1 : 2;
    }
    return p;
}

__device__ __forceinline__ double pow_planned(double x, double y, PowPlan p) {
    if (p.kind == 0) return pow(x, y);
    double r = (p.kind == 2) ? sqrt(x) : 1.0;
    for (int i = 0; i < p.n; i++) r *= x;
    return p.neg ? 1.0 / r : r;
}

// x1^y1 / x2^y2 with both exponents planned: the two magnitudes as products and square roots and
// at most one division (within a few ulp of the quotient of the pow() forms)
__device__ __forceinline__ double pow_ratio_planned(double x1, double y1, PowPlan p1, double x2, double y2,
                                                   PowPlan p2) {
    if (p1.kind == 0 || p2.kind == 0) return pow_planned(x1, y1, p1) / pow_planned(x2, y2, p2);
    double r1 = (p1.kind == 2) ? sqrt(x1) : 1.0, r2 = (p2.kind == 2) ? sqrt(x2) : 1.0;
    for (int i = 0; i < p1.n; i++) r1 *= x1;
    for (int i = 0; i < p2.n; i++) r2 *= x2;
    if (p1.neg) return p2.neg ? r2 / r1 : 1.0 / (r1 * r2);
    return p2.neg ? r1 * r2 : r1 / r2;
}

struct Dbn2plArgs {
    double sepa_init_log10, rchar, gi, go;
    int num_steps, n_freq, fobs_sorted;
    int n_mtot, n_mrat, n_redz, n_interp;
    PowPlan p_outer, p_inner;   // exponents -go + gi and gi - 1 of the hardening rate
};

// Several (mtot, mrat) cells per block (`cpb`, chosen by the host so that cpb x n_redz rows nearly
// fill the block): a cell's redshift rows alone would leave most of a warp idle (101 rows are three
// warps and five lanes), and GB300 charges an FP64 warp instruction in full however few lanes are
// active.  Row r of the block is redshift r / nc of its cell r % nc (nc cells in the block); each cell's step
// tables live in its own slice of shared memory, built by the whole block.  Each row's arithmetic is
// the single-cell kernel's.
constexpr int WALK_MAX_CELLS = 16;

__global__ void __launch_bounds__(512) k_dbn_2pwl(CyConst cc, Dbn2plArgs a, int cpb, const double *__restrict__ fobs,
                           const double *__restrict__ hard_norm, const double *__restrict__ nden,
                           const double *__restrict__ mtot, const double *__restrict__ mrat,
                           const double *__restrict__ redz, const double *__restrict__ gmt_time,
                           const double *__restrict__ zgrid_g, const double *__restrict__ agrid_g,
                           const double *__restrict__ dgrid_g, double *__restrict__ redz_final,
                           double *__restrict__ diff_num) {
    extern __shared__ double smem[];
    const int S = a.num_steps, NI = a.n_interp, NF = a.n_freq;
    const int ncell = a.n_mtot * a.n_mrat;
    const int cell0 = blockIdx.x * cpb;
    const int nc = min(cpb, ncell - cell0);   // cells of this block
    double *zg = smem;
    double *ag = zg + NI;
    double *dg = ag + NI;
    double *sz = dg + NI;            // [NI] dz/dt of each age-table interval
    double *ft = sz + NI;
    double *cells = ft + NF;         // per cell: sepa [S+1], frst [S+1], dadt [S+1], dts [S], tevo [S]
    const int per_cell = 3 * (S + 1) + 2 * S;
    __shared__ double s_fmax;
    __shared__ int s_first[WALK_MAX_CELLS];
    __shared__ double s_sqrt_mt[WALK_MAX_CELLS], s_mt3[WALK_MAX_CELLS], s_mr12[WALK_MAX_CELLS];

    for (int i = threadIdx.x; i < NI; i += blockDim.x) {
        zg[i] = zgrid_g[i];
        ag[i] = agrid_g[i];
        dg[i] = dgrid_g[i];
    }
    for (int i = threadIdx.x; i < NF; i += blockDim.x) ft[i] = fobs[i];
    __syncthreads();
    for (int i = threadIdx.x; i < NI - 1; i += blockDim.x) sz[i] = (zg[i + 1] - zg[i]) / (ag[i + 1] - ag[i]);
    if (threadIdx.x < nc) {   // log10 separation nodes by repeated subtraction, one thread per cell
        const int cell = cell0 + threadIdx.x;
        const double mt = mtot[cell / a.n_mrat];
        double *sepa = cells + (size_t)threadIdx.x * per_cell;
        const double risco = 3.0 * HGB_CY_SCHW * mt;
        const double dx = (a.sepa_init_log10 - log10(risco)) / S;
        double sl = a.sepa_init_log10;
        sepa[0] = sl;
        for (int s = 1; s <= S; s++) {
            sl -= dx;
            sepa[s] = sl;
        }
        const double mr = mrat[cell % a.n_mrat];
        s_sqrt_mt[threadIdx.x] = sqrt(mt);
        s_mt3[threadIdx.x] = pow(mt, 3.0);
        s_mr12[threadIdx.x] = pow(1.0 + mr, 2.0);
    }
    __syncthreads();
    // per node: sp^1.5 as sp sqrt(sp), the hardening model's (half-)integer powers as products
    // (pow_planned), and the GW rate with the cell's mt^3 and (1 + mr)^2 taken once: each within a
    // few ulp of the pow() forms of sam_cyutils.pyx:240-253 and holodeck/cyutils.pyx
    for (int i = threadIdx.x; i < nc * (S + 1); i += blockDim.x) {
        const int c = i / (S + 1), s = i % (S + 1), cell = cell0 + c;
        const double mr = mrat[cell % a.n_mrat], norm = hard_norm[cell];
        const double sqrt_mt = s_sqrt_mt[c], mt3 = s_mt3[c], mr12 = s_mr12[c];
        double *sepa = cells + (size_t)c * per_cell;
        double *frst = sepa + (S + 1), *dadt = frst + (S + 1);
        const double sp = pow(10.0, sepa[s]);
        sepa[s] = sp;
        frst[s] = cc.kfreq * sqrt_mt / (sp * sqrt(sp));
        const double xx = sp / a.rchar;
        double dd = -norm * pow_ratio_planned(1.0 + xx, -a.go + a.gi, a.p_outer, xx, a.gi - 1.0, a.p_inner);
        dd += cc.c_dadt * mt3 * mr / (sp * sp * sp) / mr12;
        dadt[s] = dd;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nc * S; i += blockDim.x) {
        const int c = i / S, s = i % S;
        double *sepa = cells + (size_t)c * per_cell;
        const double *dadt = sepa + 2 * (S + 1);
        double *dts = sepa + 3 * (S + 1);
        dts[s] = 2.0 * (sepa[s + 1] - sepa[s]) / (dadt[s] + dadt[s + 1]);
    }
    __syncthreads();
    // Steps that cannot bracket any target are skipped without changing a result: the observed
    // frequency of a step is at most its rest-frame frequency (z >= 0 after clamping) and at least
    // frst / (1 + z_start), because the redshift only decreases from the starting redshift.
    double fmin_all = ft[0], fmax_all = ft[0];
    for (int f = 1; f < NF; f++) {
        fmin_all = fmin_all < ft[f] ? fmin_all : ft[f];
        fmax_all = fmax_all > ft[f] ? fmax_all : ft[f];
    }
    if (threadIdx.x < nc) {   // running time and first useful step, one thread per cell
        double *sepa = cells + (size_t)threadIdx.x * per_cell;
        const double *frst = sepa + (S + 1), *dts = sepa + 3 * (S + 1);
        double *tevo = sepa + 3 * (S + 1) + S;
        double te = 0.0;
        for (int s = 0; s < S; s++) {
            te += dts[s];
            tevo[s] = te;
        }
        int first = 0;   // first step whose right edge reaches fmin
        while (first < S && frst[first + 1] < fmin_all) first++;
        s_first[threadIdx.x] = first;
        if (threadIdx.x == 0) s_fmax = fmax_all;
    }
    __syncthreads();
    const double fmax = s_fmax;

    const double age_universe = ag[NI - 1];
    for (int r = threadIdx.x; r < nc * a.n_redz; r += blockDim.x) {
        // redshift-major: a warp's lanes hold a few neighbouring redshifts of every cell of the block
        // (mostly one mtot, so one rest-frequency table), whose walks have similar lengths
        const int c = r % nc, kk = r / nc;
        const int cell = cell0 + c;
        const double *frst = cells + (size_t)c * per_cell + (S + 1);
        const double *dts = cells + (size_t)c * per_cell + 3 * (S + 1);
        const double *tevo = dts + S;
        const int s_begin = s_first[c];
        long row = ((long)cell * a.n_redz + kk);
        double *rf = redz_final + row * NF;
        double *dn = diff_num + row * NF;
        for (int f = 0; f < NF; f++) {
            rf[f] = -1.0;
            dn[f] = 0.0;
        }
        // age at the starting redshift (sam_cyutils.pyx:563-573)
        double zk = redz[kk];
        int zi = hgb::bracket_decreasing_from0(NI, zk, zg);
        if (zi > NI - 2) zi = NI - 2;
        double rage = hgb::interp_between(zk, zg[zi], zg[zi + 1], ag[zi], ag[zi + 1]);
        double gmt = gmt_time[row];
        const double fstop = fmax * (1.0 + zk) * (1.0 + 1e-12);
        int il = 0;
        int fp = 0;                 // first target >= the left frequency (targets ascending)
        bool have_prev = false;     // right edge of the previous step, reused as this step's left edge
        double prev_tr = 0.0, prev_zr = 0.0, prev_fr = 0.0;
        for (int s = s_begin; s < S; s++) {
            if (frst[s] > fstop) break;
            double time_right = tevo[s] + gmt + rage;
            double time_left, redz_left, fl;
            bool reuse = have_prev;
            have_prev = false;
            if (reuse) {
                time_left = prev_tr;
            } else {
                time_left = time_right - dts[s];
            }
            if (time_left > age_universe) continue;
            if (reuse) {
                redz_left = prev_zr;
            } else {
                il = hgb::while_while_increasing(il, NI, time_left, ag);
                redz_left = zg[il] + (time_left - ag[il]) * sz[il];
            }
            if (redz_left < 0.0) continue;
            fl = reuse ? prev_fr : frst[s] / (1.0 + redz_left);
            int ir = hgb::while_while_increasing(il, NI, time_right, ag);
            double redz_right = zg[ir] + (time_right - ag[ir]) * sz[ir];
            double zr_raw = redz_right;
            if (redz_right < 0.0) redz_right = 0.0;
            double fr = frst[s + 1] / (1.0 + redz_right);
            if (zr_raw >= 0.0) {
                have_prev = true;
                prev_tr = time_right;
                prev_zr = zr_raw;
                prev_fr = fr;
            }
            int il_step = il;
            il = ir;
            int f0;
            if (a.fobs_sorted) {
                while (fp > 0 && ft[fp - 1] >= fl) fp--;
                while (fp < NF && ft[fp] < fl) fp++;
                f0 = fp;
                if (f0 >= NF || ft[f0] > fr) continue;
            } else {
                f0 = 0;
            }
            for (int f = f0; f < NF; f++) {
                double ftarget = ft[f];
                if (ftarget < fl || fr < ftarget) {
                    if (a.fobs_sorted) break;   // ascending targets: nothing further lies inside
                    continue;
                }
                double new_time = hgb::interp_between(ftarget, fl, fr, time_left, time_right);
                if (new_time > ag[NI - 1]) break;
                // phase 1 records the bracket; k_dbn_2pwl_eval turns it into redz_final / diff_num
                rf[f] = (double)il_step;
                dn[f] = new_time;
            }
        }
    }
}

// y^p of the hardening shape's outer factor, y = 1 + x: a planned negative (half-)integer power from one
// reciprocal square root, any other exponent as pow_planned
__device__ __forceinline__ double shape_outer(double y, double p, PowPlan plan) {
    if (plan.kind == 0 || !plan.neg || !hgb::fast_range(y)) return pow_planned(y, p, plan);
    const double r = hgb::fast_rsqrt(y), r2 = r * r;
    double v = plan.kind == 2 ? r : 1.0;
    for (int i = 0; i < plan.n; i++) v *= r2;
    return v;
}

// The walk for ascending targets: which step brackets a target is decided in FP32, and only the bracket
// found is evaluated in FP64.
// One block takes a run of mrat cells of one mtot.  What depends on mtot alone (separations, rest
// frequencies, the steps' shape and GW sums alpha and beta, see k_hardening_norm_sub) is built once per
// block, and the cells' step times 1 / (norm alpha + gw_k beta) and their running sums.  Then, for a few
// cells at a time:
//   A  one thread per (cell, redshift) row walks its nodes in FP32 (time, redshift, observed frequency:
//      relative error a few 1e-7 against steps of some percent) and notes for each target the step and
//      the age-table interval it starts in;
//   B  the row's (redshift, target) elements, spread over all threads with the target fastest, test the
//      noted step in FP64 and move by one where FP32 chose a neighbour.  The tests at a node are
//      ft (1 + z) >= frst from its right and <= frst from its left with the same values, so every target
//      between the first node and the last belongs to a step.  Of the time in the bracket,
//        t_l + (t_r - t_l) (ft - f_l) / (f_r - f_l),  f = frst / (1 + z),
//      both frequencies' quotients and the interpolation's are one reciprocal: twenty FP64 operations.
// That a target lies in one step needs nodes whose frequencies and times ascend, and a time to start from.
// Where they do not (a normalisation, mass, redshift or merger time that is NaN or negative, an infinite
// step, a start inside the ISCO),
//   C  takes the row's steps one after another, as k_dbn_2pwl does: the same brackets, and a NaN where a
//      time is one.  (At the end, so that the rows' walk and search keep their registers.)
// FP64 bounds both forms, but the walk in FP64 spent some 25 operations a step on 80 steps a row,
// comparisons among them, with lanes idle where their neighbours walk longer, and wrote its outputs
// eight bytes to a line.  91 x 81 x 101 points, 40 targets: 3130 us before, 930 us now (FP64 pipe 72% busy); 30^3 points
// with 20: 443 and 141 us.
constexpr int WK_THREADS = 256;
constexpr unsigned WK_NONE = 0xFFFFFFFFu, WK_LATER = 0xFFFFFFFEu;   // no bracket; a row of C
constexpr double WK_SCALE = 0x1.0p40;   // of the FP64 frequencies, some 1e-10 Hz: keeps the bracket's products in range

struct WalkShape {
    int cb;       // cells walked together
    int qc;       // mrat cells per block
    int rows;     // rows of one pass (cb cells' rows go in passes of this many)
    size_t smem;
};

// The log10 separations of the reference's loop (S subtractions of dx, each rounded) without the chain of
// S dependent operations: while the values stay in one binade, with last place u, every rounded step is
// the same multiple of u (dx rounded to it; only a dx half way between two would alternate), so the
// nodes of a binade are first - j d exactly.  Writes the segments' first values, steps and first nodes and
// returns their number; what does not fit the scheme (values at or below 1, a tie) goes to `node`, one
// after another, as the last, empty segment's place.
constexpr int WK_SEGS = 8;

__device__ int log_nodes(double init, double dx, int S, double *first, double *step, int *seg, double *node) {
    double sl = init;
    int s = 0, k = 0;
    while (s <= S && k < WK_SEGS - 1 && sl > 1.0 && dx > 0.0) {
        const double low = __hiloint2double(__double2hiint(sl) & 0x7FF00000, 0);   // the binade's lower end
        const double d = sl - (sl - dx);
        if (!(sl - dx >= low) || 2.0 * fabs(dx - d) >= low * 0x1.0p-52) {   // one step leaves it, or a tie
            seg[k] = s;
            first[k] = sl;
            step[k++] = 0.0;
            sl -= dx;
            s++;
            continue;
        }
        int j = (int)fmin((sl - low) / d, (double)(S - s));   // steps that stay
        while (j > 0 && sl - (double)j * d < low) j--;
        while (j < S - s && sl - (double)(j + 1) * d >= low) j++;
        seg[k] = s;
        first[k] = sl;
        step[k++] = d;
        s += j + 1;
        sl = (sl - (double)j * d) - dx;   // the step out of the binade rounds by the next one's last place
    }
    seg[k] = min(s, S + 1);
    for (; s <= S; s++) {
        node[s] = sl;
        sl -= dx;
    }
    return k;
}

// One row's steps in turn, with the comparisons of k_dbn_2pwl in their order (NaN fails them all, so a step
// without a time brackets every target).  tc: time of the nodes from the first, norm al + gw be: one over
// a step's time.
__device__ __forceinline__ void walk_stepwise(const Dbn2plArgs &a, const double *ft, const double *zg, const double *ag,
                                           const double *sz, const double *frst, const double *al, const double *be,
                                           const double *tc, double norm, double gw, double zk, double rage, double gmt,
                                           double *rf, double *dn) {
    const int S = a.num_steps, NI = a.n_interp, NF = a.n_freq;
    for (int f = 0; f < NF; f++) {
        rf[f] = -1.0;
        dn[f] = 0.0;
    }
    const double fstop = ft[NF - 1] * (1.0 + zk) * (1.0 + 1e-12);
    int first = 0, il = 0;
    while (first < S && frst[first + 1] < ft[0]) first++;
    bool have_prev = false;
    double prev_tr = 0.0, prev_zr = 0.0, prev_fr = 0.0;
    for (int s = first; s < S; s++) {
        if (frst[s] > fstop) break;
        const bool reuse = have_prev;
        have_prev = false;
        const double tr = tc[s + 1] + gmt + rage;
        const double tl = reuse ? prev_tr : tr - 1.0 / __fma_rn(norm, al[s], gw * be[s]);
        if (tl > ag[NI - 1]) continue;
        double zl = prev_zr;
        if (!reuse) {
            il = hgb::while_while_increasing(il, NI, tl, ag);
            zl = zg[il] + (tl - ag[il]) * sz[il];
        }
        if (zl < 0.0) continue;
        const double fl = reuse ? prev_fr : frst[s] / (1.0 + zl);
        const int ir = hgb::while_while_increasing(il, NI, tr, ag);
        const double zr = zg[ir] + (tr - ag[ir]) * sz[ir];
        const double fr = frst[s + 1] / (1.0 + (zr < 0.0 ? 0.0 : zr));
        if (zr >= 0.0) {
            have_prev = true;
            prev_tr = tr;
            prev_zr = zr;
            prev_fr = fr;
        }
        const int il_step = il;
        il = ir;
        for (int f = 0; f < NF; f++) {
            if (ft[f] < fl || fr < ft[f]) continue;
            const double tt = hgb::interp_between(ft[f], fl, fr, tl, tr);
            if (tt > ag[NI - 1]) break;
            rf[f] = (double)il_step;
            dn[f] = tt;
        }
    }
}

// a merger time before the start or none, or no age to start from
__device__ __forceinline__ bool wk_odd_row(double gmt, double rage) {
    const float sum = hgb::f64_to_f32_rz(gmt + rage);
    return __double2hiint(gmt) < 0 || sum != sum;
}

__host__ __device__ inline int wk_stride(int nf) { return nf | 1; }   // an odd row length keeps the lanes' rows in different banks

__global__ void __launch_bounds__(WK_THREADS, 3) k_dbn_2pwl_walk(
    CyConst cc, Dbn2plArgs a, WalkShape ws, const double *__restrict__ fobs, const double *__restrict__ hard_norm,
    const double *__restrict__ mtot, const double *__restrict__ mrat, const double *__restrict__ redz,
    const double *__restrict__ gmt_time, const double *__restrict__ zgrid_g, const double *__restrict__ agrid_g,
    double *__restrict__ redz_final, double *__restrict__ diff_num) {
    extern __shared__ double smem[];
    const int S = a.num_steps, NI = a.n_interp, NF = a.n_freq, NZ = a.n_redz;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double *zg = smem, *ag = zg + NI, *sz = ag + NI;   // age table and dz/dt of its intervals
    double *ft = sz + NI;                              // [NF]
    double *rage = ft + NF;                            // [NZ] age at the starting redshift
    double *frst = rage + NZ, *al = frst + S + 1, *be = al + S + 1;   // [S + 1] nodes, [S] steps
    double *base = be + S + 1;                         // [rows] merger time
    double *tn = base + ws.rows;                       // [qc][S + 1] time of a cell's nodes from the first
    float *zgf = (float *)(tn + (size_t)ws.qc * (S + 1)), *agf = zgf + NI, *szf = agf + NI, *ftf = szf + NI;
    float *frf = ftf + NF;
    unsigned *code = (unsigned *)(frf + S + 1);   // [rows][wk_stride(NF)] step | interval << 16
    __shared__ int s_first;
    __shared__ unsigned s_odd;   // the block's cells (bit per cell) whose rows are C's
    __shared__ int s_later;      // whether C has rows
    __shared__ unsigned queue[WK_THREADS / 32][64];
    const int nqb = (a.n_mrat + ws.qc - 1) / ws.qc;
    const int ii = blockIdx.x / nqb, q0 = (blockIdx.x % nqb) * ws.qc, q1 = min(q0 + ws.qc, a.n_mrat);
    const double mt = mtot[ii];

    if (t == 0) {
        s_odd = 0u;
        s_later = 0;
    }
    for (int i = t; i < NI; i += WK_THREADS) {
        zg[i] = zgrid_g[i];
        ag[i] = agrid_g[i];
    }
    bool odd = false;   // a NaN among the targets, frequencies that do not ascend
    for (int f = t; f < NF; f += WK_THREADS) {
        const double x = fobs[f];
        ft[f] = x * WK_SCALE;
        ftf[f] = (float)x;
        odd |= (__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll) > 0x7FF0000000000000ll;
    }
    // nodes: separation, and in the steps' arrays for now the hardening shape and 1 / separation^3
    double *sepa = tn;   // the first cell's times come later
    __shared__ double s_sl[WK_SEGS], s_d[WK_SEGS];
    __shared__ int s_seg[WK_SEGS + 1], s_nseg;
    if (t == 0) s_nseg = log_nodes(a.sepa_init_log10, (a.sepa_init_log10 - log10(3.0 * HGB_CY_SCHW * mt)) / S, S, s_sl, s_d, s_seg, sepa);
    __syncthreads();
    for (int k = 0; k < s_nseg; k++)
        for (int s = s_seg[k] + t; s < s_seg[k + 1]; s += WK_THREADS) sepa[s] = __fma_rn(-(double)(s - s_seg[k]), s_d[k], s_sl[k]);
    __syncthreads();
    {
        const double inv_rchar = 1.0 / a.rchar, kf = cc.kfreq * sqrt(mt), pin = 1.0 - a.gi;
        for (int s = t; s <= S; s += WK_THREADS) {
            const double sp = exp10(sepa[s]);
            const double r = hgb::fast_range(sp) ? hgb::fast_rsqrt(sp) : 1.0 / sqrt(sp);
            const double xx = sp * inv_rchar, r2 = r * r;
            sepa[s] = sp;
            const double fr = kf * (r2 * r);
            frst[s] = fr * WK_SCALE;
            frf[s] = (float)fr;
            al[s] = shape_outer(1.0 + xx, -a.go + a.gi, a.p_outer) *
                    pow_planned(xx, pin, PowPlan{a.p_inner.kind, a.p_inner.n, !a.p_inner.neg});
            be[s] = r2 * r2 * r2;
        }
    }
    __syncthreads();
    for (int i = t; i < NI; i += WK_THREADS) {
        if (i < NI - 1) {
            sz[i] = (zg[i + 1] - zg[i]) / (ag[i + 1] - ag[i]);
            szf[i] = (float)sz[i];
        }
        zgf[i] = (float)zg[i];
        agf[i] = (float)ag[i];
    }
    for (int k = t; k < NZ; k += WK_THREADS) {   // sam_cyutils.pyx:563-573
        const double zk = redz[k];
        int zi = hgb::bracket_decreasing_from0(NI, zk, zg);
        if (zi > NI - 2) zi = NI - 2;
        rage[k] = hgb::interp_between(zk, zg[zi], zg[zi + 1], ag[zi], ag[zi + 1]);
    }
    if (t == 0) {   // first step whose right edge reaches the lowest target (z >= 0: observed <= rest frame)
        int lo = 0, hi = S;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (frst[mid + 1] < ft[0]) lo = mid + 1;
            else hi = mid;
        }
        s_first = lo;
    }
    for (int s0 = 0; s0 < S; s0 += WK_THREADS) {   // sums over a step's two nodes over twice its width
        const int s = s0 + t;
        double av = 0.0, bv = 0.0;
        if (s < S) {
            const double w = sepa[s] - sepa[s + 1];
            const double c = 0.5 * (hgb::fast_range(w) ? hgb::fast_rcp(w) : 1.0 / w);
            av = (al[s] + al[s + 1]) * c;
            bv = (be[s] + be[s + 1]) * c;
            const long long lo = __double_as_longlong(frst[s]), hi = __double_as_longlong(frst[s + 1]);
            odd |= !(lo > 0 && hi > lo && hi < 0x7FF0000000000000ll);
        }
        __syncthreads();   // every node of this run is read, and node s0 + WK_THREADS is rewritten next
        if (s < S) {
            al[s] = av;
            be[s] = bv;
        }
    }
    if (odd) atomicOr(&s_odd, ~0u);
    __syncthreads();
    const int first = s_first;
    const float age_f = (float)ag[NI - 1] * 1.000001f;   // beyond it in FP32: beyond the table's end in FP64
    const long long age_bits = __double_as_longlong(ag[NI - 1]);
    const int stride = wk_stride(NF);

    // node times of the block's cells: every step by its own thread, then one thread per cell adds them in
    // step order.  The order matters: a target reached just before the present is at z ~ 1e-7, where one
    // ulp of the time (64 s) is 1e-9 of the distance, so the sums round as the reference's do.
    const int nq = q1 - q0;
    for (int i = t; i < nq * S; i += WK_THREADS) {
        const int c = i / S, s = i % S;
        const double mr = mrat[q0 + c], opq = 1.0 + mr;
        const double gw_k = -cc.c_dadt * (mt * mt * mt) * mr / (opq * opq);
        const double y = __fma_rn(hard_norm[(long)ii * a.n_mrat + q0 + c], al[s], gw_k * be[s]);
        const bool plain = hgb::fast_range(y);   // positive and finite, as its reciprocal
        if (!plain) atomicOr(&s_odd, 1u << c);
        tn[(size_t)c * (S + 1) + s + 1] = plain ? hgb::fast_rcp(y) : 1.0 / y;
    }
    __syncthreads();
    const unsigned odd_cells = s_odd;
    if (t < nq) {
        double *tc = tn + (size_t)t * (S + 1);
        double te = 0.0;
        tc[0] = 0.0;
#pragma unroll 8
        for (int s = 1; s <= S; s++) {
            te += tc[s];
            tc[s] = te;
        }
    }

    for (int qb = q0; qb < q1; qb += ws.cb) {
        const int nc = min(ws.cb, q1 - qb);
        const long cell0 = (long)ii * a.n_mrat + qb;
        const double *tnb = tn + (size_t)(qb - q0) * (S + 1);
        for (int row0 = 0; row0 < nc * NZ; row0 += ws.rows) {
            const int nr = min(ws.rows, nc * NZ - row0);
            __syncthreads();   // node times are complete; the previous pass is written
            // ---- A
            if (t < nr) {
                const int c = (row0 + t) / NZ, kk = (row0 + t) % NZ;
                const double b = gmt_time[(cell0 + c) * NZ + kk];
                base[t] = b;
                const float bf = hgb::f64_to_f32_rz(b + rage[kk]);
                const double *tc = tnb + (size_t)c * (S + 1);
                unsigned *cd = code + t * stride;
                int f = 0;
                unsigned rest = WK_NONE;
                if (((odd_cells >> (qb - q0 + c)) & 1u) || wk_odd_row(b, rage[kk])) {
                    rest = WK_LATER;
                    s_later = 1;
                } else {
                    float tl = bf + hgb::f64_to_f32_rz(tc[first]);
                    int il = 0, hi = NI - 2;   // interval of the first node
                    while (il < hi) {
                        const int mid = (il + hi) >> 1;
                        if (agf[mid + 1] < tl) il = mid + 1;
                        else hi = mid;
                    }
                    int n = first;
                    for (; n < S && f < NF && tl <= age_f; n++) {
                        const float tr = bf + hgb::f64_to_f32_rz(tc[n + 1]), fr = frf[n + 1];
                        const int in = il;
                        while (il < NI - 2 && agf[il + 1] < tr) il++;
                        const float p = 1.0f + fmaxf(zgf[il] + (tr - agf[il]) * szf[il], 0.0f);
                        while (f < NF && ftf[f] * p < fr) cd[f++] = (unsigned)n | ((unsigned)in << 16);
                        tl = tr;
                    }
                    if (n == S && S > first) rest = (unsigned)(S - 1) | ((unsigned)il << 16);   // within FP32 of the last node
                }
                for (; f < NF; f++) cd[f] = rest;
            }
            __syncthreads();
            // ---- B
            double *rf = redz_final + (cell0 * NZ + row0) * NF;
            double *dn = diff_num + (cell0 * NZ + row0) * NF;
            auto element = [&](unsigned packed) {   // row << 16 | target
                const int r = (int)(packed >> 16), f = (int)(packed & 0xFFFFu);
                const unsigned cd = code[r * stride + f];
                double out_r = -1.0, out_t = 0.0;
                int s = (int)(cd & 0xFFFFu), il = (int)(cd >> 16);
                const double *tc = tnb + (size_t)((row0 + r) / NZ) * (S + 1);
                const double gmt = base[r], ra = rage[(row0 + r) % NZ], target = ft[f];
                for (int go = 0; go <= S; go++) {   // at most one move in practice
                    const double tl = tc[s] + gmt + ra, tr = tc[s + 1] + gmt + ra;
                    if (__double_as_longlong(tl) > age_bits) break;
                    while (il < NI - 2 && __double_as_longlong(ag[il + 1]) < __double_as_longlong(tl)) il++;
                    while (il > 0 && __double_as_longlong(ag[il]) > __double_as_longlong(tl)) il--;
                    const double zl = __fma_rn(tl - ag[il], sz[il], zg[il]);
                    if (__double2hiint(zl) < 0) break;
                    const double pl = 1.0 + zl, fl = frst[s];
                    const double x = __fma_rn(target, pl, -fl);
                    if (__double2hiint(x) < 0) {   // below the step
                        if (s == first) break;
                        s--;
                        continue;
                    }
                    int ir = il;
                    while (ir < NI - 2 && __double_as_longlong(ag[ir + 1]) < __double_as_longlong(tr)) ir++;
                    double zr = __fma_rn(tr - ag[ir], sz[ir], zg[ir]);
                    if (__double2hiint(zr) < 0) zr = 0.0;
                    const double pr = 1.0 + zr, fr = frst[s + 1];
                    const double y = __fma_rn(-target, pr, fr);
                    if (__double2hiint(y) < 0) {   // above it
                        if (s == S - 1) break;
                        s++;
                        continue;
                    }
                    const double den = __fma_rn(fr, pl, -(fl * pr));
                    const double num = (tr - tl) * x * pr;
                    const double tt = hgb::fast_range(den) ? __fma_rn(num, hgb::fast_rcp(den), tl) : tl + num / den;
                    if (!(__double_as_longlong(tt) > age_bits)) {
                        out_r = hgb::f32_to_f64_scaled((float)il, 0);   // the interval the evaluation starts from
                        out_t = tt;
                    }
                    break;
                }
                const long e = (long)r * NF + f;
                rf[e] = out_r;
                dn[e] = out_t;
            };
            const int dr = WK_THREADS / NF, df = WK_THREADS - dr * NF;
            int r = t / NF, f = t - r * NF;
            int held = 0;   // collected elements of this warp
            unsigned *q = queue[warp];
            for (int i0 = 32 * warp; i0 < nr * NF; i0 += WK_THREADS) {
                const unsigned cd = r < nr ? code[r * stride + f] : WK_NONE;
                const bool live = cd < WK_LATER;
                if (r < nr && cd == WK_NONE) {
                    const long e = (long)r * NF + f;
                    rf[e] = -1.0;
                    dn[e] = 0.0;
                }
                const unsigned m = __ballot_sync(0xffffffffu, live);
                if (live) q[held + __popc(m & ((1u << lane) - 1u))] = (unsigned)r << 16 | (unsigned)f;
                held += __popc(m);
                __syncwarp();
                if (held >= 32) {
                    element(q[lane]);
                    held -= 32;
                    const unsigned more = lane < held ? q[32 + lane] : 0u;
                    __syncwarp();
                    if (lane < held) q[lane] = more;
                    __syncwarp();
                }
                r += dr;
                f += df;
                if (f >= NF) {
                    f -= NF;
                    r++;
                }
            }
            if (lane < held) element(q[lane]);
            __syncwarp();
        }
    }
    __syncthreads();
    if (!s_later) return;
    // ---- C
    for (int i = t; i < nq * NZ; i += WK_THREADS) {
        const int c = i / NZ, kk = i % NZ;
        const long cell = (long)ii * a.n_mrat + q0 + c;
        const double b = gmt_time[cell * NZ + kk], mr = mrat[q0 + c], opq = 1.0 + mr;
        if (((odd_cells >> c) & 1u) || wk_odd_row(b, rage[kk]))
            walk_stepwise(a, ft, zg, ag, sz, frst, al, be, tn + (size_t)c * (S + 1), hard_norm[cell],
                          -cc.c_dadt * (mt * mt * mt) * mr / (opq * opq), redz[kk], rage[kk], b,
                          redz_final + (cell * NZ + kk) * NF, diff_num + (cell * NZ + kk) * NF);
    }
}

// Cells and rows of a block, and its shared memory: cells walked together fill the threads with rows, and
// a block takes up to eight of them where that leaves about eight blocks a multiprocessor.
WalkShape walk_shape(const Dbn2plArgs &a) {
    WalkShape w;
    const long cells = (long)a.n_mtot * a.n_mrat;
    w.qc = (int)std::max(1L, std::min(8L, std::min((long)a.n_mrat, hgb::ceil_div(cells, 8L * hgb::sm_count()))));
    w.cb = std::max(1, std::min(w.qc, WK_THREADS / a.n_redz));
    w.rows = std::min(WK_THREADS, w.cb * a.n_redz);
    const size_t row_bytes = sizeof(unsigned) * wk_stride(a.n_freq);
    w.rows = std::max(1, std::min<int>(w.rows, (int)(48 * 1024 / row_bytes)));
    const size_t nodes = (size_t)a.num_steps + 1;
    w.smem = sizeof(double) * (3 * (size_t)a.n_interp + a.n_freq + a.n_redz + 3 * nodes + w.rows + w.qc * nodes) +
             sizeof(float) * (3 * (size_t)a.n_interp + a.n_freq + nodes) + row_bytes * w.rows;
    return w;
}

// Phase 2 of the Fixed_Time_2PL_SAM number: every (redz, frequency) element of a (mtot, mrat) cell
// whose target was bracketed (sam_cyutils.pyx:731-768).  One block per cell.  Targets without a bracket
// come in runs, and an FP64 instruction costs a warp the same with one live lane as with 32, so each
// warp first collects its bracketed elements, and evaluates them 32 at a time.
// With the rest frequency F = f (1 + z) the separation is k13 F^(-2/3) and the GW rate gw_k / sepa^3 is
// G F^2, so one reciprocal gives the residence time (2/3) sepa / (norm shape(x) + G F^2), x = sepa / rchar;
// F^(-1/3) takes an FP32 start and one third-order step.  36 FP64 operations for the half-integer powers
// of the default model, where five quotients, two roots and their products took 75.  FP64 bounds it:
// 91 x 81 x 101 points, 40 targets: 2327 us before, 1106 us now.
constexpr int EV_WARPS = 8;

__global__ void __launch_bounds__(32 * EV_WARPS) k_dbn_2pwl_eval(CyConst cc, Dbn2plArgs a, const double *__restrict__ fobs,
                                const double *__restrict__ hard_norm, const double *__restrict__ nden,
                                const double *__restrict__ mtot, const double *__restrict__ mrat,
                                const double *__restrict__ zgrid_g, const double *__restrict__ agrid_g,
                                const double *__restrict__ dgrid_g, double *__restrict__ redz_final,
                                double *__restrict__ diff_num) {
    extern __shared__ double smem[];
    const int NI = a.n_interp, NF = a.n_freq;
    double *zg = smem;
    double *ag = zg + NI;
    double *dg = ag + NI;            // comoving distance in Mpc
    double *ft = dg + NI;
    double *sz = ft + NF;            // [NI] dz/dt and d(d_C)/dt of each age-table interval
    double *sd = sz + NI;
    __shared__ int queue[EV_WARPS][64];
    const int cell = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ii = cell / a.n_mrat, jj = cell % a.n_mrat;
    for (int i = threadIdx.x; i < NI; i += blockDim.x) {
        zg[i] = zgrid_g[i];
        ag[i] = agrid_g[i];
        dg[i] = dgrid_g[i] * (1.0 / HGB_CY_MPC) * 0x1.0p-50;   // (exact; `unit` carries the square's 2^100)
    }
    for (int i = threadIdx.x; i < NF; i += blockDim.x) ft[i] = fobs[i];
    __syncthreads();
    for (int i = threadIdx.x; i < NI - 1; i += blockDim.x) {
        const double dt = ag[i + 1] - ag[i];
        sz[i] = (zg[i + 1] - zg[i]) / dt;
        sd[i] = (dg[i + 1] - dg[i]) / dt;
    }
    __shared__ double s_k13r, s_g;
    const double mt = mtot[ii], mr = mrat[jj], norm = hard_norm[cell];
    if (threadIdx.x == 0) {
        const double k13 = cc.ksepa * pow(mt, 1.0 / 3.0), opq = 1.0 + mr;
        s_k13r = k13 / a.rchar;
        s_g = -cc.c_dadt * (mt * mt * mt) * mr / (opq * opq) / (k13 * k13 * k13);
    }
    __syncthreads();
    const double k13r = s_k13r, gw = s_g;
    const double pout = -a.go + a.gi, pin = 1.0 - a.gi;
    const PowPlan inner{a.p_inner.kind, a.p_inner.n, !a.p_inner.neg};
    // 2^100: a density near the least double (a mass function's cutoff) keeps its bits through the residence
    // time's factors, small in these units, until the distance takes the power out again
    const double unit = cc.fourpi * (2.0 / 3.0) * a.rchar * 0x1.0p100;
    const int nzf = a.n_redz * NF;
    const long base = (long)cell * nzf;

    auto element = [&](int e) {
        const double t = diff_num[base + e];
        // the bracket's first age interval, a small whole number
        int ni = (int)hgb::f64_to_f32_rz(redz_final[base + e]);
        const long long tb = __double_as_longlong(t);
        while (ni < NI - 2 && __double_as_longlong(ag[ni + 1]) < tb) ni++;
        while (ni > 0 && __double_as_longlong(ag[ni]) > tb) ni--;
        const double dt = t - ag[ni];
        const double z = __fma_rn(dt, sz[ni], zg[ni]), dcm = __fma_rn(dt, sd[ni], dg[ni]);
        const double p = 1.0 + z, F = ft[e % NF] * p;
        // F^(-1/3) = r (1 + e / 3 + 2 e^2 / 9 + ...) with e = 1 - F r^3 of a few 1e-7
        const double r0 = hgb::f32_to_f64_scaled(rcbrtf(hgb::f64_to_f32_rz(F)), 0);
        const double err = __fma_rn(-(F * r0), r0 * r0, 1.0);
        const double r = __fma_rn(r0 * err, __fma_rn(2.0 / 9.0, err, 1.0 / 3.0), r0);
        const double x = k13r * (r * r);
        const double shape = shape_outer(1.0 + x, pout, a.p_outer) * pow_planned(x, pin, inner);
        const double rate = __fma_rn(norm, shape, gw * (F * F));
        const double inv = hgb::fast_range(rate) ? hgb::fast_rcp(rate) : 1.0 / rate;
        redz_final[base + e] = z;
        diff_num[base + e] = nden[(long)cell * a.n_redz + e / NF] * (unit * x * inv) * (p * (dcm * dcm));
    };
    int held = 0;   // collected elements of this warp
    int *q = queue[warp];
    for (int e0 = 32 * warp; e0 < nzf; e0 += 32 * EV_WARPS) {
        const int e = e0 + lane;
        // without a bracket (-1) an element stays -1 / 0
        const bool live = e < nzf && __double2hiint(redz_final[base + e]) >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, live);
        if (live) q[held + __popc(m & ((1u << lane) - 1u))] = e;
        held += __popc(m);
        __syncwarp();
        if (held >= 32) {
            element(q[lane]);
            held -= 32;
            const int more = lane < held ? q[32 + lane] : 0;
            __syncwarp();
            if (lane < held) q[lane] = more;
            __syncwarp();
        }
    }
    if (lane < held) element(q[lane]);
}

// ---- FP32 production mode of k_dbn_2pwl_eval
//
// The age -> redshift inversion (bracket, interpolated redshift and comoving distance) stays FP64, as
// in the reference; the residence time and the cosmological factor are FP32.  FP64 work per element:
// the bracket offset, two interpolations and the two products with the density.  The age bracket
// compares the positive FP64 ages as integers (IEEE order of positive doubles), off the FP64 pipe.
// Ranges: the hardening rate is -(A P(x) + G / x^3) with x = sepa / rchar, A = norm and
// G = |GW_DADT_SEP_CONST| mt^3 mr / (1 + mr)^2 / rchar^3 per cell; both constants are scaled by the
// same power of two 2^-e0 (e0 the larger exponent), so the sum is a normal float wherever either term
// matters, and the residence time comes out as t_s 2^-e0.

// x^y for the planned exponents in FP32 (as pow_planned / pow_ratio_planned)
__device__ __forceinline__ float pow_planned_f32(float x, float y, PowPlan p) {
    if (p.kind == 0) return powf(x, y);
    float r = (p.kind == 2) ? sqrtf(x) : 1.0f;
    for (int i = 0; i < p.n; i++) r *= x;
    return p.neg ? __fdividef(1.0f, r) : r;
}

__device__ __forceinline__ int while_while_increasing_bits(int start, int size, double val, const double *edges) {
    const long long v = __double_as_longlong(val);   // val and edges are positive: integer order is IEEE order
    int index = start;
    while ((index < size - 2) && (__double_as_longlong(edges[index + 1]) < v)) index += 1;
    while ((index > 0) && (__double_as_longlong(edges[index]) > v)) index -= 1;
    return index;
}

__global__ void k_dbn_2pwl_eval_f32(CyConst cc, Dbn2plArgs a, const double *__restrict__ fobs,
                                    const double *__restrict__ hard_norm, const double *__restrict__ nden,
                                    const double *__restrict__ mtot, const double *__restrict__ mrat,
                                    const double *__restrict__ zgrid_g, const double *__restrict__ agrid_g,
                                    const double *__restrict__ dgrid_g, double *__restrict__ redz_final,
                                    double *__restrict__ diff_num) {
    extern __shared__ double smem[];
    const int NI = a.n_interp, NF = a.n_freq;
    double *zg = smem;
    double *ag = zg + NI;
    double *dg = ag + NI;
    double *sz = dg + NI;            // [NI] dz/dt and d(d_C)/dt of each age-table interval
    double *sd = sz + NI;
    float *ft = (float *)(sd + NI);  // [NF]
    const int cell = blockIdx.x;
    const int ii = cell / a.n_mrat, jj = cell % a.n_mrat;
    for (int i = threadIdx.x; i < NI; i += blockDim.x) {
        zg[i] = zgrid_g[i];
        ag[i] = agrid_g[i];
        dg[i] = dgrid_g[i];
    }
    for (int i = threadIdx.x; i < NF; i += blockDim.x) ft[i] = hgb::f64_to_f32_rz(fobs[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < NI - 1; i += blockDim.x) {
        const double dt = ag[i + 1] - ag[i];
        sz[i] = (zg[i + 1] - zg[i]) / dt;
        sd[i] = (dg[i + 1] - dg[i]) / dt;
    }
    __shared__ float s_k13, s_as, s_gs, s_rchar_inv;
    __shared__ int s_e0;
    if (threadIdx.x == 0) {
        const double mt = mtot[ii], mr = mrat[jj], norm = hard_norm[cell];
        const double opq = 1.0 + mr, rc = a.rchar;   // products in place of powers: one thread, the block waits
        const double gc = fabs(cc.c_dadt) * (mt * mt * mt) * mr / (opq * opq) / (rc * rc * rc);
        int ea = -100000, eg = -100000;
        if (norm > 0.0) frexp(norm, &ea);
        if (gc > 0.0) frexp(gc, &eg);
        const int e0 = ea > eg ? ea : eg;
        s_e0 = e0;
        s_as = (float)ldexp(norm, -e0);   // in [0.5, 1) or flushed to 0 when negligible
        s_gs = (float)ldexp(gc, -e0);
        s_k13 = (float)(cc.ksepa * cbrt(mt));
        s_rchar_inv = (float)(1.0 / a.rchar);
    }
    __syncthreads();
    const float k13 = s_k13, as = s_as, gs = s_gs, rchar_inv = s_rchar_inv;
    const int e0 = s_e0;
    const float fourpi = (float)cc.fourpi, inv_mpc = (float)(1.0 / HGB_CY_MPC);
    const long nzf = (long)a.n_redz * NF;
    const long base = (long)cell * nzf;
    for (long e = threadIdx.x; e < nzf; e += blockDim.x) {
        const double hint = redz_final[base + e];
        if (__double_as_longlong(hint) < 0) continue;   // no bracket (-1): stays -1 / 0
        const int f = (int)(e % NF);
        const int kk = (int)(e / NF);
        const double new_time = diff_num[base + e];
        const int ni = while_while_increasing_bits((int)hint, NI, new_time, ag);
        const double dt = new_time - ag[ni];
        const double new_redz = zg[ni] + dt * sz[ni];
        const double dcom = dg[ni] + dt * sd[ni];
        const float zp1 = 1.0f + hgb::f64_to_f32_rz(new_redz);
        const float frst = ft[f] * zp1;
        const float r = rcbrtf(frst);
        const float sp = k13 * (r * r);
        const float xx = sp * rchar_inv;
        const float pw = (a.p_outer.kind && a.p_inner.kind)
                             ? pow_planned_f32(1.0f + xx, (float)(-a.go + a.gi), a.p_outer) *
                                   pow_planned_f32(xx, (float)(1.0 - a.gi), PowPlan{a.p_inner.kind, a.p_inner.n,
                                                                                   !a.p_inner.neg})
                             : __fdividef(powf(1.0f + xx, (float)(-a.go + a.gi)), powf(xx, (float)(a.gi - 1.0)));
        const float rate = fmaf(as, pw, __fdividef(gs, xx * xx * xx));
        const float tres = __fdividef((2.0f / 3.0f) * sp, rate);        // residence time 2^e0
        const float dcm = hgb::f64_to_f32_rz(dcom) * inv_mpc;
        const float cosmo_fact = fourpi * zp1 * (dcm * dcm);
        redz_final[base + e] = new_redz;
        diff_num[base + e] = nden[(long)cell * a.n_redz + kk] * hgb::f32_to_f64_scaled(tres, -e0) *
                             hgb::f32_to_f64_scaled(cosmo_fact, 0);
    }
}

// ------------------------------------------------------------------------------------------------
// differential binary number, Hard_GW
// ------------------------------------------------------------------------------------------------

// One block per run of grid points, rows of the outputs, across cells.  For GW-driven hardening the residence time is a product of powers,
//   tres = (2/3) sepa / |da/dt| = (2/3) ksepa^4 mt^(4/3) (1 + mr)^2 / (|c_dadt| mt^3 mr) (f (1 + z))^(-8/3),
// so an element is A(cell, z) B(f) with B = f^(-8/3) taken once per block and A once per grid point:
// one FP64 product per element in place of two pow() and six divisions (on this GPU an FP64 warp
// instruction holds its pipe for 64 cycles, so those set the time).  Targets are the block's fastest
// index, so the two (M, Q, Z, F) outputs are written in contiguous runs; with one thread per grid
// point walking its targets every store of a warp touched 32 lines.  A block takes up to 256 rows, so that
// the powers of the targets and of its cells' masses are shared by many points and the per-point terms
// fill its threads, whatever the grid's shape; fewer where that would leave multiprocessors without four
// blocks.  us with one thread per point, one block per cell, and so (each with the call's launch
// and allocation): 61 x 47 x 53 points, 37 targets 5059, 121, 52; 181 x 161 x 1, one target 103, 705, 70.
// The reference stops at the first target above the ISCO frequency, so target f is empty when any
// f' <= f lies above it: the running maximum of the targets decides (products by 1 + z > 0 keep the
// order).  B and the cell's constant carry 2^-80 and 2^80, which keeps A within a few decades of the
// result.  f^(2/3) and mt^(1/3) are pow() of the rounded exponents, as in the reference: a cube root is
// nearer to the real power but 4e-15 from the reference's value once it is raised to the fourth.
constexpr int GW_ROWS = 256;    // rows of a block at most, one per thread
constexpr int GW_FREQS = 512;   // targets staged at a time
constexpr double GW_SCALE = 0x1.0p80, GW_SCALE_INV = 0x1.0p-80;

__global__ void __launch_bounds__(GW_ROWS) k_dbn_gw(CyConst cc, const double *__restrict__ fobs, int NF,
                                                    const double *__restrict__ nden, const double *__restrict__ mtot,
                                                    const double *__restrict__ mrat, int nq, int nz, long total,
                                                    int rows, const double *__restrict__ redz_prime,
                                                    const double *__restrict__ zgrid, const double *__restrict__ dgrid,
                                                    int NI, double *__restrict__ redz_final,
                                                    double *__restrict__ diff_num) {
    __shared__ double fb[GW_FREQS], ftop[GW_FREQS];   // B and the running maximum of the targets
    __shared__ double s_amp[GW_ROWS], s_z[GW_ROWS];
    __shared__ int s_cut[GW_ROWS];                    // first empty target of the staged ones
    __shared__ double s_k[GW_ROWS], s_isco[GW_ROWS];  // of the block's cells
    const int t = threadIdx.x;
    const long row0 = (long)blockIdx.x * rows;
    const int nrb = (int)(total - row0 < rows ? total - row0 : rows);
    const long cell0 = row0 / nz;
    const int z0 = (int)(row0 - cell0 * nz);
    if (t < (z0 + nrb - 1) / nz + 1) {
        const double mt = mtot[(cell0 + t) / nq], mr = mrat[(cell0 + t) % nq];
        const double ks2 = cc.ksepa * cc.ksepa, opq = 1.0 + mr;
        const double m13 = pow(mt, 1.0 / 3.0), m23 = m13 * m13;
        s_k[t] = (2.0 / 3.0) * (ks2 * ks2) * (opq * opq) / (-cc.c_dadt * mr) * (m23 * m23 / mt / mt / mt) * GW_SCALE;
        s_isco[t] = cc.kfreq * sqrt(mt) / pow(3.0 * HGB_CY_SCHW * mt, 1.5);
    }
    // the row's redshift terms: A without the cell's constant
    double rzp = -1.0, zp1 = 0.0, part = 0.0, z_third = 0.0, scale = 1.0;
    const int cell = (z0 + t) / nz;
    if (t < nrb) {
        rzp = redz_prime[row0 + t];
        if (!(rzp <= 0.0)) {
            int zi = hgb::bracket_decreasing_from0(NI, rzp, zgrid);
            if (zi > NI - 2) zi = NI - 2;
            const double dcom = hgb::interp_between(rzp, zgrid[zi], zgrid[zi + 1], dgrid[zi], dgrid[zi + 1]);
            const double dcm = dcom / HGB_CY_MPC;
            zp1 = 1.0 + rzp;
            // densities near the least double (a mass function's cutoff) are carried up, so that a small
            // factor before a large one takes none of their bits
            const double nd = nden[row0 + t];
            scale = ((unsigned)__double2hiint(nd) >> 20 & 0x7FFu) < 323u ? 0x1.0p-200 : 1.0;
            part = (scale < 1.0 ? nd * 0x1.0p200 : nd) * (cc.fourpi * zp1 * (dcm * dcm));
            z_third = cbrt(zp1);
        }
    }
    double top = -INFINITY;   // (thread 0) largest target so far
    for (int f0 = 0; f0 < NF; f0 += GW_FREQS) {
        const int nfb = min(GW_FREQS, NF - f0);
        __syncthreads();   // the previous targets are done with
        for (int f = t; f < nfb; f += GW_ROWS) {
            const double p = pow(fobs[f0 + f], 2.0 / 3.0), p2 = p * p;
            fb[f] = GW_SCALE_INV / (p2 * p2);
        }
        if (t == 0) {
            for (int f = 0; f < nfb; f++) {
                const double x = fobs[f0 + f];
                top = x > top ? x : top;
                ftop[f] = top;
            }
        }
        __syncthreads();
        if (t < nrb) {
            double amp = 0.0;
            int cut = 0;
            if (!(rzp <= 0.0)) {
                // (1 + z)^(-8/3) = cbrt(1 + z) / (1 + z)^3
                amp = part * (s_k[cell] * z_third / (zp1 * zp1 * zp1)) * scale;
                const double isco = s_isco[cell];
                int hi = nfb;   // first f with ftop[f] (1 + z) > isco
                while (cut < hi) {
                    const int mid = (cut + hi) >> 1;
                    if (ftop[mid] * zp1 > isco) hi = mid;
                    else cut = mid + 1;
                }
            }
            s_amp[t] = amp;
            s_z[t] = rzp <= 0.0 ? -1.0 : rzp;
            s_cut[t] = cut;
        }
        __syncthreads();
        double *rf = redz_final + row0 * NF + f0;
        double *dn = diff_num + row0 * NF + f0;
        const int dz = GW_ROWS / nfb, df = GW_ROWS - dz * nfb;
        int z = t / nfb, f = t - z * nfb;
        while (z < nrb) {
            const long e = (long)z * NF + f;
            rf[e] = s_z[z];
            dn[e] = f < s_cut[z] ? s_amp[z] * fb[f] : 0.0;
            z += dz;
            f += df;
            if (f >= nfb) {
                f -= nfb;
                z++;
            }
        }
    }
}

// The same root with CPW cells per warp, 32 / CPW lanes each.  The lifetime's trapezoid sum is
//   T(norm) = sum_s 1 / (norm alpha_s + beta_s),  alpha_s = (shape_s + shape_s+1) / (2 dx_s) and
//   beta_s = (gw_s + gw_s+1) / (2 dx_s)  (rates counted positive, dx_s the step's width),
// so a Brent round costs a step one multiply-add, a share of a reciprocal (fast_rcp, four steps over one
// denominator) and an addition: 3.75 FP64 operations, where v_s = norm shape_s + gw_s, their sum, the
// quotient and the addition took 14.  A lane
// keeps the alpha and beta of a run of consecutive steps in registers.  Each cell's lanes share its Brent
// state (an xor-butterfly leaves the same total in all of them); the root finding itself, one exp10 and
// some fifty uniform FP64 operations a round, is shared by the warp's CPW cells, neighbours in the grid
// that need about the same number of rounds.  A node's separation, shape and 1 / x^3 depend on the total
// mass only, so a block evaluates them once for all its cells of one mass.  The log10 separations are
// init - s dx, one rounding each.
// (Separations as products of a few shared powers of ten would save another tenth of the time, and two
// roundings that come out cubed: the norm's error doubles, 4e-17 to 9e-17, so each is its own exp10.)
// The sum's grouping moves the lifetime by about 1e-16 relative, far below the root tolerance of 1e-3,
// which the root follows unless a Brent comparison falls within that margin (checked against the
// reference at 1e-10 in log10).  FP64 bounds it.  91 x 81 cells: 2822 us with one cell per warp and a
// quotient per node and round, 841 us with four (896 and 1081 with two and one), 534 us with the nodes
// shared; general exponents (two pow() a node) 3626, 1769 and 606 us.
constexpr int NB_STEPS = 320;   // steps the kernel holds in registers
constexpr int NB_WARPS = 4;     // of a block, which shares the nodes

template <int CPW>
__global__ void __launch_bounds__(32 * NB_WARPS) k_hardening_norm_sub(CyConst cc, NormArgs a, const double *__restrict__ mtot,
                                                           const double *__restrict__ mrat, int n,
                                                           double *__restrict__ norm_log10,
                                                           double *__restrict__ norm, int *d_status) {
    constexpr int LPC = 32 / CPW, NL = NB_STEPS / LPC;   // lanes per cell, steps per lane
    __shared__ double s_x[NB_STEPS + 1], s_r[NB_STEPS + 1], s_i[NB_STEPS + 1];   // nodes
    __shared__ double s_al[NB_STEPS], s_be[NB_STEPS];                            // steps
    __shared__ unsigned s_next;
    const int S = a.nsteps, t = threadIdx.x;
    const int sub = t % LPC;
    const int own = blockIdx.x * (CPW * NB_WARPS) + t / LPC;
    const int cell = min(own, n - 1);   // the last block repeats its last cell
    const double mt = mtot[cell], mr = mrat[cell];
    const double opq = 1.0 + mr;
    const double gw_k = -cc.c_dadt * (mt * mt * mt) * mr / (opq * opq);
    double al[NL], be[NL];
    // the nodes of one total mass at a time (a block of grid cells meets one or two), for all its cells
    for (bool loaded = false;;) {
        if (t == 0) s_next = 0xFFFFFFFFu;
        __syncthreads();   // (and the previous mass's steps are read)
        const unsigned first = __reduce_min_sync(0xffffffffu, loaded ? 0xFFFFFFFFu : (unsigned)cell);
        if ((t & 31) == 0 && first != 0xFFFFFFFFu) atomicMin(&s_next, first);
        __syncthreads();
        const unsigned next = s_next;
        if (next == 0xFFFFFFFFu) break;
        const double mt_n = mtot[next];
        const double dx = (a.sepa_init_log10 - log10(3.0 * HGB_CY_SCHW * mt_n)) / S;
        const double inv_rchar = 1.0 / a.rchar, pin = 1.0 - a.gi;
        for (int s = t; s <= S; s += 32 * NB_WARPS) {
            const double x = exp10(__fma_rn(-(double)s, dx, a.sepa_init_log10));
            const double xx = x * inv_rchar, x3 = x * x * x;
            s_x[s] = x;
            s_r[s] = shape_outer(1.0 + xx, -a.go + a.gi, a.p_outer) *
                     pow_planned(xx, pin, PowPlan{a.p_inner.kind, a.p_inner.n, !a.p_inner.neg});
            s_i[s] = hgb::fast_range(x3) ? hgb::fast_rcp(x3) : 1.0 / x3;
        }
        __syncthreads();
        for (int s = t; s < S; s += 32 * NB_WARPS) {
            const double w = s_x[s] - s_x[s + 1];
            const double c = 0.5 * (hgb::fast_range(w) ? hgb::fast_rcp(w) : 1.0 / w);
            s_al[s] = (s_r[s] + s_r[s + 1]) * c;
            s_be[s] = (s_i[s] + s_i[s + 1]) * c;
        }
        __syncthreads();
        if (!loaded && __double_as_longlong(mt) == __double_as_longlong(mt_n)) {
            loaded = true;
#pragma unroll
            for (int k = 0; k < NL; k++) {
                // every LPC-th step is a lane's, so the lanes read side by side; steps beyond the last add
                // 1e-60 s
                const int s = k * LPC + sub;
                al[k] = s < S ? s_al[s] : 0.0;
                be[k] = s < S ? gw_k * s_be[s] : 1e60;
            }
        }
    }

    // Brent's method as in warp_brent, one evaluation per round; the warp goes on until its last cell is
    // done (its lanes exchange partial sums, so none leaves early)
    double xa = NORM_LOG10_LO, xb = NORM_LOG10_HI, xc = 0.0, fa = 0.0, fb = 0.0, fc = 0.0, d = 0.0, e = 0.0;
    double root = 0.0;
    bool done = false, limit = false;
    for (int round = 0; round < BRENT_MAXITER + 2; round++) {
        const double nrm = exp10(round == 0 ? xa : xb);
        double part = 0.0;
#pragma unroll
        for (int k = 0; k + 1 < NL; k += 4) {
            // four steps share a reciprocal (two, at the end of an odd half): 15 FP64 operations, not 20
            const double y0 = __fma_rn(nrm, al[k], be[k]), y1 = __fma_rn(nrm, al[k + 1], be[k + 1]);
            double num = y0 + y1, den = y0 * y1;
            if (k + 3 < NL) {
                const double y2 = __fma_rn(nrm, al[k + 2], be[k + 2]), y3 = __fma_rn(nrm, al[k + 3], be[k + 3]);
                const double d2 = y2 * y3;
                num = __fma_rn(num, d2, (y2 + y3) * den);
                den *= d2;
            }
            if (hgb::fast_range(den)) {
                part = __fma_rn(num, hgb::fast_rcp(den), part);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (k + i < NL) part += 1.0 / __fma_rn(nrm, al[k + i], be[k + i]);
            }
        }
#pragma unroll
        for (int o = LPC / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        const double fv = part - a.target_time;
        if (round == 0) {
            fa = fv;
            continue;
        }
        if (!done) {
            fb = fv;
            if (round == 1) {
                if (fa * fb > 0.0) {
                    done = true;   // no root between the ends: 0
                } else if (fa == 0.0) {
                    root = xa;
                    done = true;
                } else if (fb == 0.0) {
                    root = xb;
                    done = true;
                }
                xc = xa;
                fc = fa;
                d = xb - xa;
                e = d;
            } else if (round > BRENT_MAXITER) {
                root = xb;
                limit = done = true;
            }
        }
        if (!done) {
            if (fb * fc > 0.0) {
                xc = xa;
                fc = fa;
                d = xb - xa;
                e = d;
            }
            if (fabs(fc) < fabs(fb)) {
                xa = xb; xb = xc; xc = xa;
                fa = fb; fb = fc; fc = fa;
            }
            const double tol = 0.5 * (BRENT_XTOL + BRENT_RTOL * fabs(xb));
            const double m = 0.5 * (xc - xb);
            if (fb == 0.0 || fabs(m) < tol) {
                root = xb;
                done = true;
            } else {
                if (fabs(e) > tol && fabs(fb) < fabs(fa)) {
                    double sst;
                    if (xa == xc) {
                        sst = -fb * (xb - xa) / (fb - fa);
                    } else {
                        const double da = (fa - fb) / (xa - xb);
                        const double dc = (fc - fb) / (xc - xb);
                        sst = -fb * (fc * dc - fa * da) / (dc * da * (fc - fa));
                    }
                    if (2.0 * fabs(sst) < fmin(fabs(e), 3.0 * fabs(m) - tol)) {
                        e = d;
                        d = sst;
                    } else {
                        d = m;
                        e = m;
                    }
                } else {
                    d = m;
                    e = m;
                }
                xa = xb;
                fa = fb;
                xb = xb + ((fabs(d) > tol) ? d : ((m > 0.0) ? tol : -tol));
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
    }
    if (sub == 0 && own < n) {
        norm_log10[own] = root;
        if (norm) norm[own] = pow(10.0, root);
        if (limit) hgb::flag(d_status, HGB_STATUS_ITERATION_LIMIT);
    }
}

size_t norm_smem_per_warp(int nsteps) { return (size_t)5 * (nsteps + 1) * sizeof(double); }

}  // namespace

extern "C" {

int hgb_find_2pwl_hardening_norm(double target_time, const double *mtot, const double *mrat, int n,
                                 double sepa_init, double rchar, double gamma_inner, double gamma_outer,
                                 int nsteps, double *norm_log10, double *norm, int *d_status, void *stream) {
    HGB_CHECK_ARG(mtot && mrat && norm_log10 && n >= 0);
    HGB_CHECK_ARG(nsteps > 0 && sepa_init > 0.0 && rchar > 0.0);
    size_t per_warp = norm_smem_per_warp(nsteps);
    HGB_CHECK_ARG(per_warp <= 200 * 1024);
    if (n == 0) return HGB_OK;
    int wpb = (int)(48 * 1024 / per_warp);
    if (wpb > 4) wpb = 4;
    if (wpb < 1) wpb = 1;
    size_t smem = per_warp * wpb;
    int rc = hgb::ensure_dyn_smem((const void *)k_hardening_norm, smem);
    if (rc) return rc;
    NormArgs a{target_time, log10(sepa_init), rchar, gamma_inner, gamma_outer, nsteps,
               pow_plan(-gamma_outer + gamma_inner), pow_plan(gamma_inner - 1.0)};
    if (nsteps <= NB_STEPS) {
        cudaStream_t st = (cudaStream_t)stream;
        // four cells a warp do least work, but two spread further while their blocks leave
        // multiprocessors idle: 30 x 30 cells 174 and 128 us, 40 x 40 cells 172 and 197 us
        if (n > 2 * NB_WARPS * hgb::sm_count())
            k_hardening_norm_sub<4><<<(unsigned)hgb::ceil_div(n, 4 * NB_WARPS), 32 * NB_WARPS, 0, st>>>(
                hgb::cy_const(), a, mtot, mrat, n, norm_log10, norm, d_status);
        else
            k_hardening_norm_sub<2><<<(unsigned)hgb::ceil_div(n, 2 * NB_WARPS), 32 * NB_WARPS, 0, st>>>(
                hgb::cy_const(), a, mtot, mrat, n, norm_log10, norm, d_status);
        return hgb::check_launch();
    }
    unsigned blocks = (unsigned)hgb::ceil_div(n, wpb);
    k_hardening_norm<<<blocks, 32 * wpb, smem, (cudaStream_t)stream>>>(hgb::cy_const(), a, mtot, mrat, n,
                                                                       norm_log10, norm, d_status);
    return hgb::check_launch();
}

int hgb_dbn_2pwl_phase(const double *fobs_orb, int n_freq, int fobs_sorted, double sepa_init, int num_steps,
                       const double *hard_norm, double rchar, double gamma_inner, double gamma_outer,
                       const double *nden, const double *mtot, int n_mtot, const double *mrat, int n_mrat,
                       const double *redz, int n_redz, const double *gmt_time, const hgb_cosmo *cosmo,
                       double *redz_final, double *diff_num, int phase, void *stream) {
    HGB_CHECK_ARG(phase >= 1 && phase <= 3);
    HGB_CHECK_ARG(fobs_orb && hard_norm && mtot && mrat && cosmo && redz_final && diff_num);
    HGB_CHECK_ARG(!(phase & 1) || (redz && gmt_time));
    HGB_CHECK_ARG(!(phase & 2) || nden);
    HGB_CHECK_ARG(n_freq > 0 && num_steps > 0 && n_mtot > 0 && n_mrat > 0 && n_redz > 0);
    HGB_CHECK_ARG(cosmo->grid_size >= 2 && cosmo->grid_z && cosmo->grid_age && cosmo->grid_dcom);
    HGB_CHECK_ARG(sepa_init > 0.0 && rchar > 0.0);
    Dbn2plArgs a{log10(sepa_init), rchar, gamma_inner, gamma_outer, num_steps, n_freq, fobs_sorted ? 1 : 0,
                 n_mtot, n_mrat, n_redz, cosmo->grid_size, pow_plan(-gamma_outer + gamma_inner),
                 pow_plan(gamma_inner - 1.0)};
    unsigned blocks = (unsigned)((long)n_mtot * n_mrat);
    if (phase & 1) {
        const WalkShape ws = walk_shape(a);
        // what the walk in any order needs for one cell bounds the tables of both
        const size_t base = sizeof(double) * ((size_t)4 * cosmo->grid_size + n_freq);
        const size_t per_cell = sizeof(double) * (3 * (size_t)(num_steps + 1) + 2 * (size_t)num_steps);
        HGB_CHECK_ARG(base + per_cell <= 200 * 1024);
        // ascending targets, step and interval numbers that fit the walk's 16-bit notes, and tables that
        // fit one SM; any other call takes the FP64 walk
        if (fobs_sorted && num_steps < 0xFFFF && cosmo->grid_size < 0xFFFF && ws.smem <= 200 * 1024) {
            const int wrc = hgb::ensure_dyn_smem((const void *)k_dbn_2pwl_walk, ws.smem);
            if (wrc) return wrc;
            const unsigned wb = (unsigned)((long)n_mtot * hgb::ceil_div(n_mrat, ws.qc));
            k_dbn_2pwl_walk<<<wb, WK_THREADS, ws.smem, (cudaStream_t)stream>>>(
                hgb::cy_const(), a, ws, fobs_orb, hard_norm, mtot, mrat, redz, gmt_time, cosmo->grid_z,
                cosmo->grid_age, redz_final, diff_num);
            const int rc = hgb::check_launch();
            if (rc) return rc;
        } else {
            // cells per block: fill up to 512 rows (cpb x n_redz), within a shared-memory budget
            int cpb = 512 / n_redz;
            cpb = std::min<long>(cpb, (long)((160 * 1024 - std::min<size_t>(base, 160 * 1024)) / per_cell));
            cpb = std::max(1, std::min(cpb, WALK_MAX_CELLS));
            const size_t smem = base + per_cell * cpb;
            int src = hgb::ensure_dyn_smem((const void *)k_dbn_2pwl, smem);
            if (src) return src;
            int threads = (int)hgb::ceil_div((long)cpb * n_redz, 32) * 32;
            if (threads > 512) threads = 512;
            const unsigned wblocks = (unsigned)hgb::ceil_div((long)n_mtot * n_mrat, cpb);
            k_dbn_2pwl<<<wblocks, threads, smem, (cudaStream_t)stream>>>(hgb::cy_const(), a, cpb, fobs_orb, hard_norm, nden,
                                                                        mtot, mrat, redz, gmt_time, cosmo->grid_z,
                                                                        cosmo->grid_age, cosmo->grid_dcom, redz_final,
                                                                        diff_num);
            int rc = hgb::check_launch();
            if (rc) return rc;
        }
    }
    if (phase & 2) {
        size_t smem2 = sizeof(double) * ((size_t)5 * cosmo->grid_size + n_freq);
        if (smem2 > 48 * 1024) {
            hgb::set_cuda_error(cudaErrorInvalidValue);
            return HGB_ERR_CUDA;
        }
        const int erc = hgb::ensure_dyn_smem((const void *)k_dbn_2pwl_eval, smem2);   // beside the static queues
        if (erc) return erc;
        k_dbn_2pwl_eval<<<blocks, 256, smem2, (cudaStream_t)stream>>>(hgb::cy_const(), a, fobs_orb, hard_norm, nden,
                                                                      mtot, mrat, cosmo->grid_z, cosmo->grid_age,
                                                                      cosmo->grid_dcom, redz_final, diff_num);
        return hgb::check_launch();
    }
    return HGB_OK;
}

int hgb_dbn_2pwl_phase_f32(const double *fobs_orb, int n_freq, int fobs_sorted, double sepa_init, int num_steps,
                           const double *hard_norm, double rchar, double gamma_inner, double gamma_outer,
                           const double *nden, const double *mtot, int n_mtot, const double *mrat, int n_mrat,
                           const double *redz, int n_redz, const double *gmt_time, const hgb_cosmo *cosmo,
                           double *redz_final, double *diff_num, int phase, void *stream) {
    HGB_CHECK_ARG(phase >= 1 && phase <= 3);
    HGB_CHECK_ARG(fobs_orb && hard_norm && mtot && mrat && cosmo && redz_final && diff_num);
    HGB_CHECK_ARG(!(phase & 2) || nden);
    HGB_CHECK_ARG(n_freq > 0 && num_steps > 0 && n_mtot > 0 && n_mrat > 0 && n_redz > 0);
    HGB_CHECK_ARG(cosmo->grid_size >= 2 && cosmo->grid_z && cosmo->grid_age && cosmo->grid_dcom);
    HGB_CHECK_ARG(sepa_init > 0.0 && rchar > 0.0);
    if (phase & 1) {   // the separation-step walk is the hardening integral: FP64 in both modes
        int rc = hgb_dbn_2pwl_phase(fobs_orb, n_freq, fobs_sorted, sepa_init, num_steps, hard_norm, rchar,
                                    gamma_inner, gamma_outer, nden, mtot, n_mtot, mrat, n_mrat, redz, n_redz,
                                    gmt_time, cosmo, redz_final, diff_num, 1, stream);
        if (rc) return rc;
    }
    if (!(phase & 2)) return HGB_OK;
    Dbn2plArgs a{log10(sepa_init), rchar, gamma_inner, gamma_outer, num_steps, n_freq, fobs_sorted ? 1 : 0,
                 n_mtot, n_mrat, n_redz, cosmo->grid_size, pow_plan(-gamma_outer + gamma_inner),
                 pow_plan(gamma_inner - 1.0)};
    unsigned blocks = (unsigned)((long)n_mtot * n_mrat);
    size_t smem = sizeof(double) * (size_t)5 * cosmo->grid_size + sizeof(float) * (size_t)n_freq;
    HGB_CHECK_ARG(smem <= 48 * 1024);
    const int erc = hgb::ensure_dyn_smem((const void *)k_dbn_2pwl_eval_f32, smem);   // beside the static words
    if (erc) return erc;
    k_dbn_2pwl_eval_f32<<<blocks, 256, smem, (cudaStream_t)stream>>>(hgb::cy_const(), a, fobs_orb, hard_norm, nden,
                                                                     mtot, mrat, cosmo->grid_z, cosmo->grid_age,
                                                                     cosmo->grid_dcom, redz_final, diff_num);
    return hgb::check_launch();
}

int hgb_dbn_2pwl(const double *fobs_orb, int n_freq, int fobs_sorted, double sepa_init, int num_steps,
                 const double *hard_norm, double rchar, double gamma_inner, double gamma_outer,
                 const double *nden, const double *mtot, int n_mtot, const double *mrat, int n_mrat,
                 const double *redz, int n_redz, const double *gmt_time, const hgb_cosmo *cosmo,
                 double *redz_final, double *diff_num, void *stream) {
    return hgb_dbn_2pwl_phase(fobs_orb, n_freq, fobs_sorted, sepa_init, num_steps, hard_norm, rchar, gamma_inner,
                              gamma_outer, nden, mtot, n_mtot, mrat, n_mrat, redz, n_redz, gmt_time, cosmo,
                              redz_final, diff_num, 3, stream);
}

int hgb_dbn_gw(const double *fobs_orb, int n_freq, const double *nden, const double *mtot, int n_mtot,
               const double *mrat, int n_mrat, int n_redz, const double *redz_prime, const hgb_cosmo *cosmo,
               double *redz_final, double *diff_num, void *stream) {
    HGB_CHECK_ARG(fobs_orb && nden && mtot && mrat && redz_prime && cosmo && redz_final && diff_num);
    HGB_CHECK_ARG(n_freq > 0 && n_mtot > 0 && n_mrat > 0 && n_redz > 0);
    HGB_CHECK_ARG(cosmo->grid_size >= 2 && cosmo->grid_z && cosmo->grid_dcom);
    const long total = (long)n_mtot * n_mrat * n_redz;
    long rows = hgb::ceil_div(total, 4L * hgb::sm_count());
    if (rows > 32) rows = std::min((rows + 31) / 32 * 32, (long)GW_ROWS);   // whole warps of points
    k_dbn_gw<<<(unsigned)hgb::ceil_div(total, rows), GW_ROWS, 0, (cudaStream_t)stream>>>(
        hgb::cy_const(), fobs_orb, n_freq, nden, mtot, mrat, n_mrat, n_redz, total, (int)rows, redz_prime, cosmo->grid_z,
        cosmo->grid_dcom, cosmo->grid_size, redz_final, diff_num);
    return hgb::check_launch();
}

}  // extern "C"
