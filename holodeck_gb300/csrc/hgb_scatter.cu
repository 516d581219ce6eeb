// M-Mbulge scatter of the binary density (holodeck/sams/sam.py:1291-1394, add_scatter_to_masses),
// one redshift slice per batch entry, on the geometry prepared by hgb_scatter_plan_build:
//   1. k_gradients: per-point gradients of the slice's density by the minimum-norm-network method
//      (Nielson 1983; the gradient estimate behind scipy's CloughTocher2DInterpolator): Gauss-Seidel
//      sweeps in point order, each point's 2x2 normal system solved with its precomputed inverse,
//      until the largest relative change of a sweep falls below `grad_tol`.  One block per slice.
//      k_gradients_ph keeps several sweeps in flight on the plan's phases; k_gradients takes a plan
//      without phases, one wavefront level at a time (a level's points update concurrently and read
//      exactly the neighbour values that a sequential sweep would read).
//   2. k_clough_tocher: the C1 piecewise-cubic Clough-Tocher interpolant (centroid split) at every
//      node of the regular (log m1, log m2) grid; NaN outside the hull; NaN or negative values are
//      replaced by the value of the nearest point.
//   3. k_back_dot: the Gaussian redistribution W^T (W^T G) as the reference computes it (see
//      hgb_add_scatter_to_masses) followed by the bilinear interpolation back to the points, fused
//      into one dot product per (point, slice) with the plan's per-point row of (W W).
// FP64 throughout; built with -fmad=false (where multiply-adds are fused, explicitly).
#include <math.h>

#include <algorithm>

#include "hgb_common.cuh"

namespace {

// ---- 1. gradients
__global__ void k_gradients(hgb_scatter_plan P, const double *__restrict__ dens, int nz, double *__restrict__ vals,
                            double *__restrict__ grads, int *d_status) {
    const int z = blockIdx.x;
    const int n = P.n_mtot * P.n_mrat;
    double *f = vals + (long)z * n;
    double *g = grads + 2L * z * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        f[i] = dens[(long)i * nz + z];
        g[2 * i] = 0.0;
        g[2 * i + 1] = 0.0;
    }
    __shared__ double s_err[32];
    __syncthreads();
    bool converged = false;
    for (int it = 0; it < P.grad_maxiter; it++) {
        double err = 0.0;
        for (int lev = 0; lev < P.n_levels; lev++) {
            const int e0 = P.level_ptr[lev], e1 = P.level_ptr[lev + 1];
            for (int idx = e0 + threadIdx.x; idx < e1; idx += blockDim.x) {
                const int i = P.level_vtx[idx];
                const double fi = f[i];
                double sx = 0.0, sy = 0.0;
                for (int p = P.nbr_ptr[i]; p < P.nbr_ptr[i + 1]; p++) {
                    const int j = P.nbr_idx[p];
                    const double ex = P.nbr_w[4 * p], ey = P.nbr_w[4 * p + 1];
                    const double c = 6.0 * (f[j] - fi) - 2.0 * (g[2 * j] * ex + g[2 * j + 1] * ey);
                    sx += c * P.nbr_w[4 * p + 2];
                    sy += c * P.nbr_w[4 * p + 3];
                }
                const double *qi = P.vtx_qinv + 4 * i;
                const double nx = qi[0] * sx + qi[1] * sy;
                const double ny = qi[2] * sx + qi[3] * sy;
                double change = fmax(fabs(nx - g[2 * i]), fabs(ny - g[2 * i + 1]));
                change /= fmax(1.0, fmax(fabs(nx), fabs(ny)));
                err = fmax(err, change);
                g[2 * i] = nx;
                g[2 * i + 1] = ny;
            }
            __syncthreads();
        }
        // block-wide maximum of the sweep's relative change
        for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
        if ((threadIdx.x & 31) == 0) s_err[threadIdx.x >> 5] = err;
        __syncthreads();
        if (threadIdx.x < 32) {
            double e = (threadIdx.x < (blockDim.x >> 5)) ? s_err[threadIdx.x] : 0.0;
            for (int o = 16; o > 0; o >>= 1) e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
            if (threadIdx.x == 0) s_err[0] = e;
        }
        __syncthreads();
        converged = s_err[0] < P.grad_tol;
        __syncthreads();
        if (converged) break;
    }
    if (!converged && threadIdx.x == 0) hgb::flag(d_status, HGB_STATUS_GRADIENT_NOT_CONVERGED);
}

// The same solve with several sweeps in flight.  A sweep's levels are a chain (441 levels of about 17
// points at 91 x 81), and one level at a time leaves the SM waiting: GB300's FP64 units charge a warp
// instruction 64 cycles however few of its lanes are live, so a level of 17 points costs what 32 cost,
// on one sub-partition.  A point of sweep k + 1 needs its higher-indexed neighbours' sweep k only, and
// no neighbour lies more than D levels away, so sweep k + 1 may follow D + 1 = n_phases levels behind
// sweep k (81 levels at 91 x 81, set by the hull's fan points: five to six sweeps in flight).  The plan
// groups the points by level modulo n_phases; a pass over the phases advances every point by one
// sweep, one barrier per phase, in place:
//   * a lower-indexed neighbour (at most D levels before) has made the same sweep and not the next;
//   * a higher-indexed one (at most D levels after) has made the previous sweep and not this one;
//   * two neighbours never share a phase.
// The values that a point reads, and so the iterates, are those of sweeps one after another.
// Every update is also kept by sweep (`hist`, a ring of the sweeps in flight), since a sweep is known
// to have converged only when its last level is done and the next sweeps have begun by then; the
// converged sweep is taken from there.
// The update itself is linear in the neighbours' gradients, g_i = c_i + sum_j M_ij g_j: c_i (the
// slice's values, k_scatter_rhs) is taken once per solve and M_ij (geometry) comes with the plan, so a
// neighbour costs 4 fused multiply-adds instead of 6 and the 2x2 solve is gone.  Rounding differs
// from k_gradients by regrouping only.
// Two lanes per point, one per component, 16 points per warp, or four, a component's neighbours halved.  A point with more than HGB_SCATTER_DEG
// neighbours (the hull's fans, up to 82) takes a warp: 16 lane pairs share its neighbours.  The static
// entries of a warp's points in the next phase are loaded while the current phase computes.
// A phase is bound by its fullest sub-partitions: 90 points of about 6 neighbours are 6 warps of 13 to 15
// FP64 instructions, two warps on two of the four, 1900 cycles in a row, then the reduction and the barrier
// (ncu: the FP64 pipes of the multiprocessors that hold a slice are 39% busy).  91 x 81 points, 101 slices: 4283 us one level at a
// time, 1896 us with sweeps in flight (and 69 us for c); 181 x 161, 201 slices, where the slice exceeds
// shared memory and its gradients stay in L2: 78.5 and 13.0 ms.  There the loads are the longer chain
// and the second wave of blocks costs as much as the first, so with more slices than multiprocessors
// (AHEAD off) two blocks of 128 registers share one and no entries are loaded ahead: 16.8 ms with, 201
// slices, and 13.0 without, 304 slices 18.4 and 13.6; 152 slices 9.3 and 12.2.
// most warps of a block, by registers: two sets of entries of eight neighbours take 200 a thread
__host__ __device__ constexpr int ph_warps(bool ahead, int split) { return ahead && split == 2 ? 16 : 8; }
constexpr int PH_RING = 16;    // sweeps whose test is open (at most HGB_SCATTER_STAGES + 1)
constexpr int PH_DEG = HGB_SCATTER_DEG;

// c_i = Q_i^-1 sum_j 6 (f_j - f_i) w23_ij, by position; also the slice's values, (Z, points)
__global__ void __launch_bounds__(256) k_scatter_rhs(hgb_scatter_plan P, const double *__restrict__ dens, int nz,
                                                     double *__restrict__ vals, double2 *__restrict__ cvec) {
    const int n = P.n_mtot * P.n_mrat;
    const int p = blockIdx.x * 8 + threadIdx.y, z = blockIdx.y * 32 + threadIdx.x;
    if (p >= n || z >= nz) return;
    const int i = P.ph_info[4 * p];
    const double fi = dens[(long)i * nz + z];
    double sx = 0.0, sy = 0.0;
    for (int e = P.nbr_ptr[i]; e < P.nbr_ptr[i + 1]; e++) {
        const double c = 6.0 * (dens[(long)P.nbr_idx[e] * nz + z] - fi);
        sx = __fma_rn(c, P.nbr_w[4 * e + 2], sx);
        sy = __fma_rn(c, P.nbr_w[4 * e + 3], sy);
    }
    const double *q = P.vtx_qinv + 4 * i;
    vals[(long)z * n + i] = fi;
    cvec[(long)z * n + p] = make_double2(__fma_rn(q[1], sy, q[0] * sx), __fma_rn(q[3], sy, q[2] * sx));
}

template <int SPLIT>
struct PhPre {   // a lane's point (16 / SPLIT per warp) and its part of the row of M
    int4 info;   // point, stage, neighbours (-1: no point), first entry
    int nbr[PH_DEG / SPLIT];
    double2 m[PH_DEG / SPLIT];
    double c;
};

// lane's point of chunk `base` of a phase (points with few neighbours): what ph_entries needs
template <int SPLIT>
__device__ __forceinline__ int4 ph_point(const hgb_scatter_plan &P, const int4 ph, int base, int lane) {
    const int q = base + lane / (2 * SPLIT);
    return q < ph.z ? __ldg((const int4 *)P.ph_info + ph.x + q) : make_int4(0, 0, -1, 0);
}

template <int SPLIT>
__device__ __forceinline__ void ph_entries(const hgb_scatter_plan &P, const int4 ph, int base, int lane,
                                           const double *cz, PhPre<SPLIT> &x) {
    if (x.info.z < 0) return;
    const int part = (lane >> 1) & (SPLIT - 1);
    x.c = part ? 0.0 : __ldg(cz + 2 * (ph.x + base + lane / (2 * SPLIT)) + (lane & 1));
#pragma unroll
    for (int e = 0; e < PH_DEG / SPLIT; e++) {
        if (SPLIT * e + part < x.info.z) {
            const long k = x.info.w + (long)(SPLIT * e + part) * ph.z;
            x.nbr[e] = __ldg(P.ph_nbr + k);
            x.m[e] = __ldg((const double2 *)(P.ph_m + 4 * k + 2 * (lane & 1)));
        }
    }
}

// whether a point's change (the pair of lanes hold its components) reaches tol relative to
// max(1, |new value|).  Decided in FP32 unless within 1e-5 of the tolerance or out of FP32's range.
__device__ __forceinline__ bool ph_over(double d, double v, double tol, float tolf) {
    float cd = fabsf(hgb::f64_to_f32_rz(d)), sc = fabsf(hgb::f64_to_f32_rz(v));
    cd = fmaxf(cd, __shfl_xor_sync(0xffffffffu, cd, 1));
    sc = fmaxf(1.0f, fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 1)));
    const bool under = cd < tolf * 0.99999f * sc;
    bool over = cd >= tolf * 1.00001f * sc && cd < 1e38f && sc < 1e38f;
    if (__any_sync(0xffffffffu, !under && !over)) {
        const double dd = __shfl_xor_sync(0xffffffffu, d, 1), vv = __shfl_xor_sync(0xffffffffu, v, 1);
        if (!under && !over) {
            const double change = fmax(fabs(d), fabs(dd));
            over = change / fmax(1.0, fmax(fabs(v), fabs(vv))) >= tol;
        }
    }
    return over;
}

template <bool SMEM, bool AHEAD, int SPLIT>
__global__ void __launch_bounds__(32 * ph_warps(AHEAD, SPLIT), AHEAD ? 1 : 2) k_gradients_ph(hgb_scatter_plan P, int nz,
                                                                  const double *__restrict__ cvec,
                                                                  double *__restrict__ hist, double *grads,
                                                                  int *d_status) {
    extern __shared__ double2 sm2[];
    __shared__ int s_over[PH_RING];
    const int z = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    const int n = P.n_mtot * P.n_mrat;
    const int nph = P.n_phases, last_phase = (P.n_levels - 1) % nph, last_stage = (P.n_levels - 1) / nph;
    const int nring = last_stage + 1;   // a sweep's ring entry is rewritten once its last level is done
    int4 *ptr = (int4 *)sm2;            // [nph] the phases
    // gradients by position, advanced in place: in shared memory, or in this slice's part of `grads`
    // (read and written by this block only, a barrier apart; rewritten by point at the end)
    double *g = SMEM ? (double *)(sm2 + nph) : grads + 2L * z * n;
    const double *cz = cvec + 2L * z * n;
    const float tolf = (float)P.grad_tol;
    for (int f = t; f < nph; f += blockDim.x) ptr[f] = __ldg((const int4 *)P.ph_ptr + f);
    for (int p = t; p < n; p += blockDim.x) ((double2 *)g)[p] = make_double2(0.0, 0.0);
    if (t < PH_RING) s_over[t] = 0;
    __syncthreads();
    // prefetch: a warp's points two phases ahead (one without AHEAD), their entries one phase ahead
    constexpr int PPW = 16 / SPLIT;   // points per warp
    const int base0 = PPW * warp, part = (lane >> 1) & (SPLIT - 1);
    PhPre<SPLIT> nxt;
    nxt.info = ph_point<SPLIT>(P, ptr[0], base0, lane);
    if (AHEAD) ph_entries<SPLIT>(P, ptr[0], base0, lane, cz, nxt);
    int f1 = nph > 1 ? 1 : 0;   // the next phase
    int4 info1 = ph_point<SPLIT>(P, ptr[f1], base0, lane);
    bool converged = false;
    int k_end = -1;
    for (int T = 0; k_end < 0; T++) {
        if (t == 0) s_over[(T + 1) & (PH_RING - 1)] = 0;   // sweep T + 1 starts after this pass
        for (int phase = 0; phase < nph; phase++) {
            const int4 now = ptr[phase];
            if (!AHEAD) ph_entries<SPLIT>(P, now, base0, lane, cz, nxt);
            const PhPre<SPLIT> cur = nxt;
            nxt.info = info1;
            if (AHEAD) ph_entries<SPLIT>(P, ptr[f1], base0, lane, cz, nxt);
            f1 = f1 + 1 < nph ? f1 + 1 : 0;
            info1 = ph_point<SPLIT>(P, ptr[f1], base0, lane);
            for (int base = base0; base < now.z; base += PPW * nw) {
                PhPre<SPLIT> x;
                if (base == base0) {
                    x = cur;
                } else {
                    x.info = ph_point<SPLIT>(P, now, base, lane);
                    ph_entries<SPLIT>(P, now, base, lane, cz, x);
                }
                const int k = T - x.info.y;
                const bool live = x.info.z >= 0 && k >= 0 && k < P.grad_maxiter;
                double v = 0.0, d = 0.0;
                if (live) {
                    v = x.c;
#pragma unroll
                    for (int e = 0; e < PH_DEG / SPLIT; e++) {
                        if (SPLIT * e + part < x.info.z) {
                            const double2 gj = ((const double2 *)g)[x.nbr[e]];
                            v = __fma_rn(x.m[e].x, gj.x, v);
                            v = __fma_rn(x.m[e].y, gj.y, v);
                        }
                    }
                }
                if (SPLIT == 2) v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (live && part == 0) {
                    const int o = 2 * (now.x + base + lane / (2 * SPLIT)) + (lane & 1);
                    d = v - g[o];
                    g[o] = v;
                    hist[2L * n * ((long)z * nring + k % nring) + o] = v;
                }
                if (ph_over(d, v, P.grad_tol, tolf)) s_over[k & (PH_RING - 1)] = 1;
            }
            // points with many neighbours, one warp each, from the last warp down
            for (int q = now.z + (nw - 1 - warp); q < now.y; q += nw) {
                const int p = now.x + q;
                const int4 info = __ldg((const int4 *)P.ph_info + p);
                const int k = T - info.y;
                if (k < 0 || k >= P.grad_maxiter) continue;
                double v = lane < 2 ? cz[2 * p + lane] : 0.0, d = 0.0;
                for (int e = lane >> 1; e < info.z; e += 16) {
                    const long kk = info.w + e;
                    const double2 m = __ldg((const double2 *)(P.ph_m + 4 * kk + 2 * (lane & 1)));
                    const double2 gj = ((const double2 *)g)[__ldg(P.ph_nbr + kk)];
                    v = __fma_rn(m.x, gj.x, v);
                    v = __fma_rn(m.y, gj.y, v);
                }
#pragma unroll
                for (int o = 16; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane < 2) {
                    d = v - g[2 * p + lane];
                    g[2 * p + lane] = v;
                    hist[2L * n * ((long)z * nring + k % nring) + 2 * p + lane] = v;
                }
                if (ph_over(d, v, P.grad_tol, tolf) && lane < 2) s_over[k & (PH_RING - 1)] = 1;
            }
            __syncthreads();
            if (phase == last_phase && T >= last_stage) {   // sweep T - last_stage is complete
                const int k = T - last_stage;
                converged = s_over[k & (PH_RING - 1)] == 0;
                if (converged || k + 1 >= P.grad_maxiter) {
                    k_end = k;
                    break;
                }
            }
        }
    }
    if (!converged && t == 0) hgb::flag(d_status, HGB_STATUS_GRADIENT_NOT_CONVERGED);
    const double2 *h = (const double2 *)(hist + 2L * n * ((long)z * nring + k_end % nring));
    for (int p = t; p < n; p += blockDim.x) ((double2 *)(grads + 2L * z * n))[P.ph_info[4 * p]] = h[p];
}

size_t gradients_smem(const hgb_scatter_plan &P, bool grads) {
    return sizeof(double2) * ((size_t)P.n_phases + (grads ? (size_t)P.n_mtot * P.n_mrat : 0));
}

// ---- 2. Clough-Tocher interpolation at the regular grid's nodes.  The interpolant is linear in the
// triangle's three values and gradients, so a node's value is nine products with weights that depend
// on the geometry only.  ct_weights derives them from the Bernstein ordinates of the centroid split
// (edge ordinates ee, ordinates al towards the centroid, gam and the centre by C1 continuity, beta
// across each edge with the plan's kappa): the chain rule from the ordinates' basis values back to
// f_i, g_i.
struct CtWeights {
    int v[3];
    double f[3], x[3], y[3];   // of f_v, and of the gradient's components at v
};

__device__ __forceinline__ void ct_weights(const hgb_scatter_plan &P, int r, const double *lam, CtWeights &w) {
    double px[3], py[3], kap[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        w.v[k] = P.tri[3 * r + k];
        px[k] = P.pts[2 * w.v[k]];
        py[k] = P.pts[2 * w.v[k] + 1];
        kap[k] = P.tri_kappa[3 * r + k];
        w.f[k] = w.x[k] = w.y[k] = 0.0;
    }
    const double cx = (px[0] + px[1] + px[2]) / 3.0, cy = (py[0] + py[1] + py[2]) / 3.0;
    // micro-triangle (P_i, P_j, centroid) opposite the smallest barycentric coordinate k
    int k = 0;
    if (lam[1] < lam[k]) k = 1;
    if (lam[2] < lam[k]) k = 2;
    const int i = (k + 1) % 3, j = (k + 2) % 3;
    const double lk = k == 0 ? lam[0] : k == 1 ? lam[1] : lam[2];
    const double a = (i == 0 ? lam[0] : i == 1 ? lam[1] : lam[2]) - lk;
    const double b = (j == 0 ? lam[0] : j == 1 ? lam[1] : lam[2]) - lk;
    const double c = 3.0 * lk;
    const double a2 = a * a, b2 = b * b, c2 = c * c;
    // basis values: gam_m, al_m, beta_m, and ee of the edge (i, j)
    const double cen = c2 * c / 3.0;
    double cg[3], ca[3], cb[3];
#pragma unroll
    for (int m = 0; m < 3; m++) {
        cg[m] = cen + (m == i ? 3.0 * a * c2 : 0.0) + (m == j ? 3.0 * b * c2 : 0.0);
        ca[m] = cg[m] / 3.0 + (m == i ? 3.0 * a2 * c : 0.0) + (m == j ? 3.0 * b2 * c : 0.0);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) cb[m] = (cg[(m + 1) % 3] + cg[(m + 2) % 3]) / 3.0 + (m == k ? 6.0 * a * b * c : 0.0);
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const int p = (m + 1) % 3, q = (m + 2) % 3;   // the edge opposite m
        // beta_m = (1/4 - 3k/2) ee_pq + (1/4 + 3k/2) ee_qp + (al_p + al_q) / 2 - (1/4 - k/2) f_p - (1/4 + k/2) f_q
        const double half = 0.5 * cb[m], kc = kap[m] * cb[m];
        double epq = 0.25 * cb[m] - 1.5 * kc, eqp = 0.25 * cb[m] + 1.5 * kc;
        w.f[p] += 0.5 * kc - 0.25 * cb[m];
        w.f[q] -= 0.5 * kc + 0.25 * cb[m];
        ca[p] += half;
        ca[q] += half;
        if (m == k) {
            epq += 3.0 * a2 * b;   // p = i, q = j
            eqp += 3.0 * a * b2;
            w.f[p] += a2 * a;
            w.f[q] += b2 * b;
        }
        // ee_pq = f_p + g_p . (P_q - P_p) / 3
        const double dx = (px[q] - px[p]) / 3.0, dy = (py[q] - py[p]) / 3.0;
        w.f[p] += epq;
        w.x[p] += epq * dx;
        w.y[p] += epq * dy;
        w.f[q] += eqp;
        w.x[q] -= eqp * dx;
        w.y[q] -= eqp * dy;
    }
#pragma unroll
    for (int m = 0; m < 3; m++) {   // al_m = f_m + g_m . (C - P_m) / 3
        w.f[m] += ca[m];
        w.x[m] += ca[m] * (cx - px[m]) / 3.0;
        w.y[m] += ca[m] * (cy - py[m]) / 3.0;
    }
}

// One warp takes 32 nodes of one row (b fixed, a along the lanes) and walks a run of slices: the
// weights once, then nine multiply-adds a slice; a node outside the hull (about seven in eight) copies
// its nearest point.  The grid is written as (Z, b, a), the layout of the next kernel's rows, with each
// run's largest exponent beside it (gexp, CT_NOSKIP where a value is negative, infinite or NaN).  With
// the ordinates formed again for every slice and the lanes along b (stores 8 N bytes apart) the stage
// took 1457 us at 91 x 81 x 101, 169 us now; 10.4 and 1.3 ms at 181 x 161 x 201.
constexpr int CT_ROWS = 8;             // warps per block
constexpr int CT_SLICES = 26;          // slices per warp at most: the weights cost about as much as 16 slices
constexpr unsigned CT_NOSKIP = 0x7FFu;

__global__ void __launch_bounds__(32 * CT_ROWS) k_clough_tocher(hgb_scatter_plan P, int nz, int zper,
                                                                const double *__restrict__ vals,
                                                                const double *__restrict__ grads,
                                                                double *__restrict__ grid,
                                                                unsigned short *__restrict__ gexp) {
    const int N = P.n_grid, n = P.n_mtot * P.n_mrat, nc = (N + 31) / 32;
    const int lane = threadIdx.x & 31;
    const long unit = (long)blockIdx.x * CT_ROWS + (threadIdx.x >> 5);   // (row, run of 32 nodes)
    if (unit >= (long)N * nc) return;
    const int b = (int)(unit / nc), c = (int)(unit % nc), a = 32 * c + lane;
    const bool in = a < N;
    int r = -1, near = 0;
    CtWeights w;
    if (in) {
        const long src = (long)a * N + b;
        r = P.grid_tri[src];
        near = P.grid_near[src];
        if (r >= 0) {
            const double lam[3] = {P.grid_bary[3 * src], P.grid_bary[3 * src + 1], P.grid_bary[3 * src + 2]};
            ct_weights(P, r, lam, w);
        }
    }
    const int z0 = blockIdx.y * zper, z1 = min(z0 + zper, nz);
    for (int z = z0; z < z1; z++) {
        const double *f = vals + (long)z * n;
        double val = 0.0;
        if (in) {
            bool bad = true;
            if (r >= 0) {
                const double2 *g = (const double2 *)grads + (long)z * n;
                val = 0.0;
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    const double2 gm = g[w.v[m]];
                    val = __fma_rn(w.f[m], f[w.v[m]], val);
                    val = __fma_rn(w.x[m], gm.x, val);
                    val = __fma_rn(w.y[m], gm.y, val);
                }
                // NaN or negative (an FP64 comparison costs as much as a product; the bits decide)
                const unsigned hi = (unsigned)__double2hiint(val), lo = (unsigned)__double2loint(val);
                const unsigned ah = hi & 0x7FFFFFFFu;
                bad = ah > 0x7FF00000u || (ah == 0x7FF00000u && lo) || ((hi >> 31) && (ah | lo));
            }
            if (bad) val = f[near];   // sam.py:1367-1376
            grid[((long)z * N + b) * N + a] = val;
        }
        const unsigned hi = (unsigned)__double2hiint(val), lo = (unsigned)__double2loint(val);
        const bool negative = (hi >> 31) && ((hi & 0x7FFFFFFFu) | lo);
        const unsigned e = __reduce_max_sync(0xffffffffu, negative ? CT_NOSKIP : (hi >> 20) & 0x7FFu);
        if (lane == 0) gexp[((long)z * N + b) * nc + c] = (unsigned short)e;
    }
}

// ---- 3+4. redistribution and bilinear interpolation back to the points, as one dot product per
// (point, slice): out = sum_j bw_i[j] ((1 - ty) G[j][b] + ty G[j][b + 1]), with the two weight rows
// (1 - ty) bw_i and ty bw_i precomputed, two fused multiply-adds per element.  One block per point,
// four slices per warp, the lanes along j.
// Every term is positive and the Gaussian weights span hundreds of decades, so most of a row cannot
// reach the sum's last bit: a run of 32 elements is passed over where its largest weight times its
// largest value, times 32, lies 2^-66 below a lower bound of the sum (the largest over all runs of
// smallest weight times largest value).  What is passed over adds up to less than 2^-59 of the sum,
// 1/64 of half an ulp.  At the default grid and scatter half the runs remain (a quarter at 0.1 dex,
// three quarters at 0.6).  Rows with a negative, infinite or NaN value are summed in full.
// FP64 bounds it: 1391 us at 91 x 81 x 101 with every run and a five-step reduction per output,
// 651 us now; 15.8 and 9.5 ms at 181 x 161 x 201.
constexpr int BD_WARPS = 8, BD_SLICES = 4;

__global__ void __launch_bounds__(32 * BD_WARPS) k_back_dot(hgb_scatter_plan P, const double *__restrict__ gridT,
                                                            const unsigned short *__restrict__ gexp, int nz,
                                                            bool skip, double *__restrict__ dens) {
    extern __shared__ double sw[];   // [2][N] the point's weight rows, then [2][nc] their exponents (min, max)
    const int N = P.n_grid, nc = (N + 31) / 32;
    short2 *swe = (short2 *)(sw + 2 * N);
    const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = P.back_idx[2 * i + 1];
    const double *w = P.back_w + 2L * i * N;
    for (int u = warp; skip && u < 2 * nc; u += BD_WARPS) {
        const int row = u >= nc, j = 32 * (row ? u - nc : u) + lane;
        const double x = j < N ? w[row * N + j] : 0.0;
        if (j < N) sw[row * N + j] = x;
        const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7FFu;
        const unsigned top = __reduce_max_sync(0xffffffffu, j < N ? e : 0u);
        const unsigned low = __reduce_min_sync(0xffffffffu, j < N ? e : 0x7FFu);
        if (lane == 0) swe[u] = make_short2((short)low, (short)top);
    }
    __syncthreads();
    if (skip) w = sw;
    for (int z0 = BD_SLICES * warp; z0 < nz; z0 += BD_SLICES * BD_WARPS) {
        // lane: (slice, row) pair lane % 8, runs lane / 8, lane / 8 + 4, ...; need: bit per run to sum
        unsigned need = 0xFFFFFFFFu;
        if (skip) {
            const int sl = (lane & 7) >> 1, row = lane & 1, z = z0 + sl;
            int low = -100000;
            bool full = false;
            const unsigned short *ge = gexp + ((long)min(z, nz - 1) * N + b + row) * nc;
            for (int c = lane >> 3; c < nc; c += 4) {
                const int e = ge[c], el = swe[row * nc + c].x;
                full = full || e == (int)CT_NOSKIP;
                if (e > 0 && el > 0) low = max(low, el + e);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                if (o == 2 || o == 4) continue;   // the slice's lanes: both rows, all runs
                low = max(low, __shfl_xor_sync(0xffffffffu, low, o));
                full = full | (bool)__shfl_xor_sync(0xffffffffu, (int)full, o);
            }
            need = 0u;
            for (int c = lane >> 3; c < nc; c += 4)
                if (full || swe[row * nc + c].y + ge[c] + 2 + 5 > low - 66) need |= 1u << c;
            need |= __shfl_xor_sync(0xffffffffu, need, 8);
            need |= __shfl_xor_sync(0xffffffffu, need, 16);
        }
        unsigned m[BD_SLICES][2];
        unsigned any = 0u;
#pragma unroll
        for (int s = 0; s < BD_SLICES; s++)
#pragma unroll
            for (int row = 0; row < 2; row++) {
                const unsigned x = __shfl_sync(0xffffffffu, need, 2 * s + row);
                m[s][row] = z0 + s < nz ? x : 0u;
                any |= m[s][row];
            }
        double acc[BD_SLICES] = {};
        const double *g0 = gridT + ((long)z0 * N + b) * N;
        for (int c = 0; c < nc; c++) {
            const unsigned bit = skip ? 1u << c : 0xFFFFFFFFu;
            const int j = 32 * c + lane;
            if (!(any & bit) || j >= N) continue;
            const double w0 = w[j], w1 = w[N + j];
#pragma unroll
            for (int s = 0; s < BD_SLICES; s++) {
                const double *g = g0 + (long)s * N * N + j;
                if (m[s][0] & bit) acc[s] = __fma_rn(w0, g[0], acc[s]);
                if (m[s][1] & bit) acc[s] = __fma_rn(w1, g[N], acc[s]);
            }
        }
        // four sums over 32 lanes: the first two steps halve the sums a lane carries, six additions in all
        const bool h1 = lane & 16, h2 = lane & 8;
        const double p0 = (h1 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, h1 ? acc[0] : acc[2], 16);
        const double p1 = (h1 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, h1 ? acc[1] : acc[3], 16);
        double v = (h2 ? p1 : p0) + __shfl_xor_sync(0xffffffffu, h2 ? p0 : p1, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int z = z0 + (lane >> 3);   // lanes 0, 8, 16, 24 hold slices 0 .. 3
        if ((lane & 7) == 0 && z < nz) dens[(long)i * nz + z] = v;
    }
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" {

size_t hgb_scatter_workspace_bytes(int n_mtot, int n_mrat, int n_redz, int n_grid) {
    if (n_mtot < 2 || n_mrat < 2 || n_redz < 1 || n_grid < 2) return 0;
    size_t n = (size_t)n_mtot * n_mrat, NN = (size_t)n_grid * n_grid;
    const size_t last = std::max(NN, 2 * HGB_SCATTER_STAGES * n);   // the regular grid; the sweeps in flight
    return align256(sizeof(double) * n * n_redz) + 2 * align256(sizeof(double) * 2 * n * n_redz) +
           align256(sizeof(double) * last * n_redz) +
           align256(sizeof(short) * n_grid * (((size_t)n_grid + 31) / 32) * n_redz) + 16;   // the base, rounded up
}

int hgb_add_scatter_to_masses(const hgb_scatter_plan *plan, double *dens, int n_redz, void *workspace,
                              size_t workspace_bytes, int *d_status, void *stream) {
    HGB_CHECK_ARG(plan && dens && n_redz >= 1);
    const hgb_scatter_plan &P = *plan;
    HGB_CHECK_ARG(P.n_mtot >= 2 && P.n_mrat >= 2 && P.n_grid >= 2 && P.n_levels >= 1);
    HGB_CHECK_ARG(P.pts && P.tri && P.tri_kappa && P.vtx_qinv && P.nbr_ptr && P.nbr_idx && P.nbr_w);
    HGB_CHECK_ARG(P.level_ptr && P.level_vtx && P.grid_tri && P.grid_bary && P.grid_near);
    HGB_CHECK_ARG(P.back_idx && P.back_t && P.back_w && P.grad_maxiter >= 1);
    size_t need = hgb_scatter_workspace_bytes(P.n_mtot, P.n_mrat, n_redz, P.n_grid);
    if (!workspace || workspace_bytes < need) return HGB_ERR_WORKSPACE;
    const size_t n = (size_t)P.n_mtot * P.n_mrat, NN = (size_t)P.n_grid * P.n_grid;
    char *w = (char *)(((uintptr_t)workspace + 15) & ~(uintptr_t)15);   // pairs of doubles are read whole
    double *vals = (double *)w;
    w += align256(sizeof(double) * n * n_redz);
    double *grads = (double *)w;
    w += align256(sizeof(double) * 2 * n * n_redz);
    double *cvec = (double *)w;
    w += align256(sizeof(double) * 2 * n * n_redz);
    double *gridA = (double *)w;
    double *hist = gridA;   // the sweeps in flight are done with before the grid is written
    w += align256(sizeof(double) * std::max(NN, 2 * HGB_SCATTER_STAGES * n) * n_redz);
    unsigned short *gexp = (unsigned short *)w;
    cudaStream_t st = (cudaStream_t)stream;

    int rc, dev = 0, smem_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // the phases where the plan has them and their table fits one SM; the gradients beside it where
    // they fit too (grids up to about 14000 points)
    const bool aligned = (((uintptr_t)P.ph_ptr | (uintptr_t)P.ph_info | (uintptr_t)P.ph_m) & 15) == 0;   // rows of 16 bytes
    if (P.ph_ptr && P.ph_info && P.ph_nbr && P.ph_m && aligned && P.n_phases >= 1 && P.phase_width >= 1 &&
        gradients_smem(P, false) + 1024 <= (size_t)smem_optin) {
        HGB_CHECK_ARG((P.n_levels - 1) / P.n_phases < HGB_SCATTER_STAGES);
        k_scatter_rhs<<<dim3((unsigned)hgb::ceil_div((long)n, 8), (unsigned)hgb::ceil_div(n_redz, 32)), dim3(32, 8), 0,
                        st>>>(P, dens, n_redz, vals, (double2 *)cvec);
        if ((rc = hgb::check_launch())) return rc;
        const bool in_smem = gradients_smem(P, true) + 1024 <= (size_t)smem_optin;
        const size_t smem = gradients_smem(P, in_smem);
        // more slices than multiprocessors, outside shared memory: two blocks side by side hide each
        // other's loads, and no second wave remains
        const bool ahead = in_smem || n_redz <= hgb::sm_count();
        // Four lanes a point instead of two halve the chain of a phase and add some work: the faster form
        // while a phase leaves FP64 units idle (us with two and with four lanes: 30x30 points, 30 to a
        // phase, 538 and 445; 50x45 878 and 822; 61x57 1111 and 1124; 91x81 1899 and 2032; the line lies between
        // phases of 56 points, 1801 and 1721 on other values, and of 58, 1869 and 1885) and outside
        // shared memory, where loads make the chain (181x161 points, 152 slices: 9.3 and 8.6 ms), unless
        // two blocks fill the FP64 units, which the walk beside them needs (201 slices: 13.0 and 12.8,
        // but the whole call is 0.4% longer)
        const int split = (in_smem ? P.phase_width <= 56 : ahead) ? 2 : 1;
        // the widest phase's points and a warp for a fan point, whole sub-partitions
        int nw = (int)hgb::ceil_div(P.phase_width, 16 / split) + 1;
        nw = std::min(ph_warps(ahead, split), (nw + 3) / 4 * 4);
        const auto fn = !in_smem ? (ahead ? k_gradients_ph<false, true, 2> : k_gradients_ph<false, false, 1>)
                        : split == 1 ? k_gradients_ph<true, true, 1> : k_gradients_ph<true, true, 2>;
        if ((rc = hgb::ensure_dyn_smem((const void *)fn, smem))) return rc;
        fn<<<n_redz, 32 * nw, smem, st>>>(P, n_redz, cvec, hist, grads, d_status);
    } else {
        k_gradients<<<n_redz, 256, 0, st>>>(P, dens, n_redz, vals, grads, d_status);
    }
    if ((rc = hgb::check_launch())) return rc;
    const int N = P.n_grid, nc = (N + 31) / 32;
    const int zparts = (int)hgb::ceil_div(n_redz, CT_SLICES), zper = (int)hgb::ceil_div(n_redz, zparts);
    const dim3 gct((unsigned)hgb::ceil_div((long)N * nc, CT_ROWS), (unsigned)zparts);
    k_clough_tocher<<<gct, 32 * CT_ROWS, 0, st>>>(P, n_redz, zper, vals, grads, gridA, gexp);
    if ((rc = hgb::check_launch())) return rc;
    // a bit per run of 32 nodes: rows of up to 1024 (grids of up to 256 edges along mtot) stage their
    // weights and pass runs over, longer ones are summed in full
    const bool skip = nc <= 32;
    const size_t bd_smem = skip ? sizeof(double) * 2 * N + sizeof(short2) * 2 * nc : 0;
    k_back_dot<<<(unsigned)n, 32 * BD_WARPS, bd_smem, st>>>(P, gridA, gexp, n_redz, skip, dens);
    return hgb::check_launch();
}

}  // extern "C"
