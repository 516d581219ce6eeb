// Cell integration and per-bin strain on the (M-1, Q-1, Z-1, F) bin grid (kernel k_cells):
//  * NUMBER: integrate_differential_number_3dx1d (holodeck/sams/sam_cyutils.pyx:115-216)
//  * STRAIN: char_strain_sq_from_bin_edges_redz (holodeck/gravwaves.py:694-724)
//  * both in one pass for gwb() (sam.py:930-935): each vertex of dnum and redz_final is read by the four
//    (mtot, mrat) cells that share it, and number / h2fdf are written once.
// One block, or a few, per (mtot, mrat) cell, the frequency fastest over its threads.  Built with -fmad=false: the
// eight-vertex sum and the midpoints round like the Cython/numpy code; the strain product is regrouped
// (see bin_strain), which moves it by a few ulp.
#include <limits.h>
#include <math.h>
#include <stdlib.h>

#include <algorithm>

#include "hgb_common.cuh"

namespace {

struct BinGeom {
    int nm, nq, nz, nf;   // edge counts of mtot, mrat, redz; number of frequencies
};

__device__ __forceinline__ long vtx(const BinGeom &g, int m, int q, int z, int f) {
    return (((long)m * g.nq + q) * g.nz + z) * g.nf + f;
}

struct StrainArgs {
    double gw_src_const;
    const double *dc_val, *dc_der;
    const double2 *dc_cub;   // [dc_n][2] cubic coefficients (may be null)
    int dc_n, dc_log2;       // dc_log2: log2 of a power of two dc_n up to 2^20, -1 otherwise
    double dc_h;             // 1 / dc_n
};

StrainArgs strain_args(double k, const hgb_cosmo *c) {
    const bool pairs = ((uintptr_t)c->dc_cub & 15) == 0;   // else as without the table
    StrainArgs s{k, c->dc_val, c->dc_der, pairs ? (const double2 *)c->dc_cub : nullptr, c->dc_n, -1, 1.0 / c->dc_n};
    if ((c->dc_n & (c->dc_n - 1)) == 0 && c->dc_n <= (1 << 20)) {
        s.dc_log2 = 0;
        while ((1 << s.dc_log2) < c->dc_n) s.dc_log2++;
    }
    return s;
}

// Comoving distance at y = 1 + z > 1.  u = y^(-1/2) is an FP32 estimate with one FP64 Newton step, as in
// comoving_distance_fast and with its bits (near z = 0 the distance is the small 1 - u, so another
// rounding there would show); the interval comes from u's bits, its cubic from the table.
__device__ __forceinline__ double distance_at(const StrainArgs &s, double y) {
    const float u0f = rsqrtf(hgb::f64_to_f32_rn_normal(y));
    const double u0 = hgb::f32_to_f64_scaled(u0f, 0), half = hgb::f32_to_f64_scaled(u0f, -1);
    const double u = half * (3.0 - y * (u0 * u0));
    // k = floor(u 2^L), at most 2^L - 1, from the bits of u in (0, 1 + 1e-14)
    const unsigned hi = (unsigned)__double2hiint(u);
    const int sh = 1023 - (int)(hi >> 20) - s.dc_log2;   // u 2^L = 1.m 2^-sh
    int k = sh > 0 ? 0 : (int)(((hi & 0xFFFFFu) | 0x100000u) >> (20 + sh));
    k = min(k, s.dc_n - 1);
    const double t = __fma_rn(u, (double)s.dc_n, -hgb::f32_to_f64_scaled((float)k, 0));   // exact product
    const double2 c01 = __ldg(s.dc_cub + 2 * k), c23 = __ldg(s.dc_cub + 2 * k + 1);
    return __fma_rn(__fma_rn(__fma_rn(c23.y, t, c23.x), t, c01.y), t, c01.x);
}

// gravwaves.py:694-724 on a bin with midpoint redshift z > 0, y = 1 + z, rearranged:
// hs = K mc (2 mc fr)^(2/3) / dc with fr = fc y is [K mc (2 mc)^(2/3) fc^(2/3)] y^(2/3) / dc, the first
// factor (amp) once per (mtot, mrat) cell and frequency.  y^(2/3) = y y^(-1/3), an FP32 cube root with one
// third-order step.
__device__ __forceinline__ double bin_strain(const StrainArgs &s, double z, double y, double amp, double fc_df) {
    const bool table = s.dc_cub && s.dc_log2 >= 0 && __double2hiint(y) < (1023 + 100) << 20;   // an infinite z: as before
    const double dc = table ? distance_at(s, y) : hgb::comoving_distance_fast(s.dc_val, s.dc_der, s.dc_n, s.dc_h, z);
    const double r0 = hgb::f32_to_f64_scaled(rcbrtf(hgb::f64_to_f32_rz(y)), 0);
    const double yr = y * r0;
    const double e = __fma_rn(-yr, r0 * r0, 1.0);   // 1 - y r0^3, a few 1e-7
    const double y23 = __fma_rn(yr * e, __fma_rn(2.0 / 9.0, e, 1.0 / 3.0), yr);
    const double inv = hgb::fast_range(dc) ? hgb::fast_rcp(dc) : 1.0 / dc;
    const double hs = amp * y23 * inv;
    return (hs * hs) * fc_df;
}

// One block, or a few, per (mtot, mrat) bin cell (cell_split).  A thread keeps one frequency (the threads' fastest index, so a
// warp's loads and stores are contiguous) and walks a run of redshifts, taking each vertex plane's values
// from memory once:
//   * the eight-vertex sum of the number keeps the reference's order, bit for bit;
//   * the strain's midpoints are taken along mtot, then mrat, then redz; halving is exact, so the sums
//     of a plane serve both of its bins and 1 + zb is one multiply-add.
// The sentinel and sign tests read the values' bits: an FP64 comparison holds the pipe as long as a
// product.  9 and 26 FP64 operations an element where 16 and some 55 were, and FP64 bounds it.
// 67 x 59 x 83 edges, 37 frequencies: number 305 us before, 263 us now, strain 1593 and 504 us;
// both together (gwb), 41 x 31 x 37, 20 frequencies: 148 and 67 us.
constexpr int CELL_THREADS = 512;       // of a block, at most
constexpr int CELL_F32_THREADS = 288;   // of an FP32 block: more leave an SM fewer warps (51 registers)
constexpr int CELL_FREQS = 256;     // frequencies side by side, at most
constexpr int STRAIN_MAX_FREQ = 3072;   // that the strain's entry points take

// How a cell's (redshift bin, frequency) elements are shared out: `fb` frequencies side by side, runs of
// `zlen` redshift bins, blockDim / fb runs a block and `parts` blocks a cell.
struct CellSplit {
    int fb, zlen, threads, parts;
};

// A warp's instruction costs the FP64 pipe the same with one live lane as with 32, and a run pays for the
// plane below its first bin (a third of a bin's work), so the runs of a block minimise warps times steps;
// of splits within 1% the one nearest to 128 threads.  With 256 threads whatever the counts, 129 to 255
// frequencies left up to half of them idle and 257 took a second walk for one; number and strain together in
// FP64 and in FP32, us before and now, redshifts in three bins of four: 91x81x101 edges, 129 frequencies 6892
// and 6199, 1704 and 1408; 40 frequencies 2033 and 1854, 497 and 425; 5 frequencies 358 and 323, 112 and 82;
// 60^3, 200 2760 and 2748, 703 and 626; 181x161x201, 100 38982 and 35723, 8976 and 8725.
// Cells that leave multiprocessors short of 16 warps are shared by several blocks, down to runs of 8 (3x3
// cells of 299 redshift bins, 129 frequencies, the whole call in FP64: 739 and 126).
CellSplit cell_split(int nf, int nzb, long cells, int threads) {
    CellSplit c;
    const int passes = (nf + CELL_FREQS - 1) / CELL_FREQS;
    c.fb = (nf + passes - 1) / passes;
    const int most = std::min(threads / c.fb, nzb);
    auto cost = [&](int runs) { return (c.fb * runs + 31) / 32 * ((nzb + runs - 1) / runs + 0.33); };
    const int step = std::max(1, most / 32);   // (a short search)
    double best = cost(1);
    for (int r = most; r > 1; r -= step) best = std::min(best, cost(r));
    int runs = 1, off = INT_MAX;
    for (int r = most; r >= 1; r = r == 1 ? 0 : std::max(1, r - step)) {
        const int d = std::abs((c.fb * r + 31) / 32 * 32 - 128);
        if (cost(r) <= 1.01 * best && d < off) {
            runs = r;
            off = d;
        }
    }
    c.zlen = (nzb + runs - 1) / runs;
    runs = (nzb + c.zlen - 1) / c.zlen;
    c.threads = (c.fb * runs + 31) / 32 * 32;
    runs = c.threads / c.fb;   // a small fb may leave room for more
    const long warps = cells * (c.threads / 32);
    const long want = std::min(hgb::ceil_div(16L * hgb::sm_count(), warps), hgb::ceil_div(c.zlen, 8L));
    if (want > 1) c.zlen = (int)hgb::ceil_div(c.zlen, want);
    c.parts = (int)hgb::ceil_div(nzb, (long)runs * c.zlen);
    return c;
}

template <bool NUMBER, bool STRAIN>
__global__ void __launch_bounds__(CELL_THREADS) k_cells(BinGeom g, CellSplit sp, StrainArgs s, const double *__restrict__ mtot, const double *__restrict__ log10_mtot,
                        const double *__restrict__ mrat, const double *__restrict__ redz,
                        const double *__restrict__ fedges, const double *__restrict__ dln_freq,
                        const double *__restrict__ dnum, const double *__restrict__ redz_final,
                        double *__restrict__ number, double *__restrict__ h2fdf, int *d_status) {
    const int cell = blockIdx.x;
    const int m = cell / (g.nq - 1), q = cell % (g.nq - 1);
    const int fb = sp.fb, runs = blockDim.x / fb;
    const int nzb = g.nz - 1, run = threadIdx.x / fb;
    const int z0 = (blockIdx.y * runs + run) * sp.zlen, z1 = min(z0 + sp.zlen, nzb);
    __shared__ double amp_mq;
    if (STRAIN) {
        if (threadIdx.x == 0) {
            // K mc (2 mc)^(2/3) with mc^(5/3) = mt^(5/3) mr / (1 + mr)^2
            const double mt = 0.5 * (mtot[m + 1] + mtot[m]);
            const double mr = 0.5 * (mrat[q + 1] + mrat[q]);
            const double c = cbrt(mt), opq = 1.0 + mr;
            amp_mq = s.gw_src_const * 1.5874010519681994748 * (mt * (c * c) * mr / (opq * opq));   // 2^(2/3)
            // the fractional powers of a negative ratio or chirp mass are NaN
            if (mr < 0.0 || (mt < 0.0 && mr > 0.0)) amp_mq = NAN;
        }
        __syncthreads();
    }
    if (run >= runs || z0 >= z1) return;
    double dmdq = 0.0;
    if (NUMBER) dmdq = (log10_mtot[m + 1] - log10_mtot[m]) * (mrat[q + 1] - mrat[q]);
    const long plane = (long)g.nq * g.nz * g.nf, row = (long)g.nz * g.nf;   // steps along mtot, mrat
    bool bad = false;
    for (int f = threadIdx.x - run * fb; f < g.nf; f += fb) {
        double amp = 0.0, fc_df = 0.0, dlnf8 = 0.0;
        if (STRAIN) {
            const double fc = 0.5 * (fedges[f + 1] + fedges[f]);
            const double c = cbrt(fc);
            amp = fc < 0.0 ? NAN : amp_mq * (c * c);
            fc_df = fc / (fedges[f + 1] - fedges[f]);
        }
        if (NUMBER) dlnf8 = dln_freq[f] * 0.125;
        double n00 = 0.0, n01 = 0.0, n10 = 0.0, n11 = 0.0, below = 0.0;   // the lower plane's values, its redshift sum
        for (int z = z0; z <= z1; z++) {
            const long v = vtx(g, m, q, z, f);
            const long out = ((long)cell * nzb + (z - 1)) * g.nf + f;
            const bool bin = z > z0;   // vertex z closes bin z - 1
            if (NUMBER) {
                const double u00 = dnum[v], u01 = dnum[v + row], u10 = dnum[v + plane], u11 = dnum[v + plane + row];
                if (bin) {   // sam_cyutils.pyx:199-214; the division by 8 is exact wherever it is taken
                    const double sum = ((((((n00 + u00) + n01) + u01) + n10) + u10) + n11) + u11;
                    const double vol = dmdq * (redz[z] - redz[z - 1]);
                    number[out] = sum * vol * dlnf8;
                }
                n00 = u00; n01 = u01; n10 = u10; n11 = u11;
            }
            if (STRAIN) {
                const double r00 = redz_final[v], r01 = redz_final[v + row];
                const double r10 = redz_final[v + plane], r11 = redz_final[v + plane + row];
                const long long b4[4] = {__double_as_longlong(r00), __double_as_longlong(r01),
                                         __double_as_longlong(r10), __double_as_longlong(r11)};
#pragma unroll
                for (int c = 0; c < 4; c++)   // below 0 and not -1 (and no -0, no NaN)
                    bad |= b4[c] < 0 && b4[c] != hgb::F64_MINUS_ONE_BITS && b4[c] != (long long)0x8000000000000000ull &&
                           (unsigned long long)b4[c] <= 0xFFF0000000000000ull;
                const double above = (r11 + r01) + (r10 + r00);
                if (bin) {
                    const double sum = above + below;   // 8 zb
                    const long long bits = __double_as_longlong(sum);
                    // zb <= 0 or NaN: infinite comoving distance, zero strain
                    h2fdf[out] = (bits > 0 && bits <= 0x7FF0000000000000ll)
                                     ? bin_strain(s, 0.125 * sum, __fma_rn(0.125, sum, 1.0), amp, fc_df) : 0.0;
                }
                below = above;
            }
        }
    }
    if (STRAIN && bad) hgb::flag(d_status, HGB_STATUS_INVALID_REDSHIFT);
}

// ---- FP32 production mode of k_cells<true, true>
//
// The same quantities from the same FP64 arrays, with FP32 arithmetic (explicit fmaf only; the file
// is built without contraction).  Values enter and leave FP32 through the integer conversions of
// hgb_common.cuh.  Scaling keeps every intermediate a normal float:
//   hs = A_mq A_f (1 + zb)^(2/3) / d_C with A_mq = K mc (2 mc)^(2/3) / D_H per cell and A_f = fc^(2/3),
//   each stored as a mantissa in [1, 2) and a power-of-two exponent (ka, kf); d_C / D_H = (1 - u) g(u)
//   from the FP32 table of hgb_cosmo; h2fdf = (hs_s^2 fc/df) 2^(2 (ka + kf)), hs_s the product of the
//   mantissas.
// A thread walks a run of redshifts at one frequency as in k_cells: half the loads and conversions of a
// thread per element, the same sums.  91x81x101 edges, 40 frequencies: 627 us before, 425 us now;
// 181x161x201, 100 frequencies: 11.4 and 8.2 ms (issue bounds it, some 60% of it conversions and tests).
struct StrainArgs32 {
    const float *g_val, *g_der;
    int n;
    float h;   // 1 / n
};

// d_C / D_H at z > 0: u = (1 + z)^(-1/2), 1 - u = z / (s (s + 1)) with s = sqrt(1 + z) (no cancellation
// as z -> 0), g(u) by cubic Hermite interpolation.
__device__ __forceinline__ float dc_over_dh_f32(const StrainArgs32 &s, float z) {
    const float sq = sqrtf(1.0f + z);
    const float u = __fdividef(1.0f, sq);
    const float w = __fdividef(z, sq * (sq + 1.0f));
    const float x = u * (float)s.n;
    int k = (int)x;
    if (k >= s.n) k = s.n - 1;
    if (k < 0) k = 0;
    const float t = x - (float)k;
    const float t2 = t * t, t3 = t2 * t;
    const float h00 = fmaf(2.0f, t3, fmaf(-3.0f, t2, 1.0f));
    const float h10 = fmaf(-2.0f, t2, t3) + t;
    const float h01 = fmaf(-2.0f, t3, 3.0f * t2);
    const float h11 = t3 - t2;
    const float gk = s.g_val[k], gk1 = s.g_val[k + 1];
    const float dk = s.g_der[k] * s.h, dk1 = s.g_der[k + 1] * s.h;
    const float g = fmaf(h00, gk, fmaf(h10, dk, fmaf(h01, gk1, h11 * dk1)));
    return w * g;
}

constexpr int F32_MAX_FREQ = 256;   // per-frequency terms staged in shared memory, a thread for each
static_assert(F32_MAX_FREQ <= CELL_FREQS, "every frequency has a thread");

__global__ void __launch_bounds__(CELL_F32_THREADS) k_cells_f32(BinGeom g, CellSplit sp, StrainArgs32 s, double amp_scale, const double *__restrict__ mtot,
                            const double *__restrict__ log10_mtot, const double *__restrict__ mrat,
                            const double *__restrict__ redz, const double *__restrict__ fedges,
                            const double *__restrict__ dln_freq, const double *__restrict__ dnum,
                            const double *__restrict__ redz_final, double *__restrict__ number,
                            double *__restrict__ h2fdf, int *d_status) {
    __shared__ float s_amp_f[F32_MAX_FREQ], s_fcdf[F32_MAX_FREQ], s_dlnf[F32_MAX_FREQ];
    __shared__ int s_kf[F32_MAX_FREQ];
    extern __shared__ float s_vol[];   // [nz - 1] dlog10M dq dz / 8 of the cell's bins
    __shared__ float s_amp_mq;
    __shared__ int s_ka;
    const int cell = blockIdx.x;
    const int m = cell / (g.nq - 1), q = cell % (g.nq - 1);
    for (int f = threadIdx.x; f < g.nf; f += blockDim.x) {
        const double fc = 0.5 * (fedges[f + 1] + fedges[f]);
        const double df = fedges[f + 1] - fedges[f];
        const float af = powf(hgb::f64_to_f32_rz(fc), 2.0f / 3.0f);   // 1e-10 .. 1e-4 Hz: a normal float
        int kf;
        const float mant = 2.0f * frexpf(af, &kf);                // af = mant 2^(kf - 1), mant in [1, 2)
        s_amp_f[f] = mant;
        s_kf[f] = kf - 1;
        s_fcdf[f] = hgb::f64_to_f32_rz(fc) / hgb::f64_to_f32_rz(df);
        s_dlnf[f] = hgb::f64_to_f32_rz(dln_freq[f]);
    }
    const double dm = log10_mtot[m + 1] - log10_mtot[m];
    const double dmdq = dm * (mrat[q + 1] - mrat[q]);
    for (int z = threadIdx.x; z < g.nz - 1; z += blockDim.x)
        s_vol[z] = hgb::f64_to_f32_rz(dmdq * (redz[z + 1] - redz[z])) * 0.125f;
    if (threadIdx.x == 0) {
        // K mc (2 mc)^(2/3) = K 2^(2/3) mc^(5/3) with mc^(5/3) = mt^(5/3) mr / (1 + mr)^2 for the chirp
        // mass mc = mt mr^(3/5) / (1 + mr)^(6/5): one cube root instead of three powers on the one
        // thread the block waits for
        const double mt = 0.5 * (mtot[m + 1] + mtot[m]);
        const double mr = 0.5 * (mrat[q + 1] + mrat[q]);
        const double c = cbrt(mt), opq = 1.0 + mr;
        const double mc53 = mt * (c * c) * mr / (opq * opq);
        int ka;
        const double mant = 2.0 * frexp(amp_scale * 1.5874010519681994 * mc53, &ka);   // 2^(2/3)
        s_amp_mq = (float)mant;
        s_ka = ka - 1;
    }
    __syncthreads();
    const float amp_mq = s_amp_mq;
    const int ka = s_ka;
    const int fb = sp.fb, runs = blockDim.x / fb;    // every frequency side by side
    const int nzb = g.nz - 1, run = threadIdx.x / fb, f = threadIdx.x - run * fb;
    const int z0 = (blockIdx.y * runs + run) * sp.zlen, z1 = min(z0 + sp.zlen, nzb);
    if (run >= runs || z0 >= z1) return;
    const float amp_f = s_amp_f[f], fcdf = s_fcdf[f], dlnf = s_dlnf[f];
    const int e2 = 2 * (ka + s_kf[f]);
    const long plane = (long)g.nq * g.nz * g.nf, row = (long)g.nz * g.nf;   // steps along mtot, mrat
    float n00 = 0.0f, n01 = 0.0f, n10 = 0.0f, n11 = 0.0f, below = 0.0f;     // the lower plane's values
    long long l00 = 0, l01 = 0, l10 = 0, l11 = 0;
    int below_sent = 0;
    bool bad = false;
    for (int z = z0; z <= z1; z++) {
        const long v = vtx(g, m, q, z, f);
        const double d00 = dnum[v], d01 = dnum[v + row], d10 = dnum[v + plane], d11 = dnum[v + plane + row];
        const long long b00 = __double_as_longlong(redz_final[v]), b01 = __double_as_longlong(redz_final[v + row]);
        const long long b10 = __double_as_longlong(redz_final[v + plane]);
        const long long b11 = __double_as_longlong(redz_final[v + plane + row]);
        const float u00 = hgb::f64_to_f32_rz(d00), u01 = hgb::f64_to_f32_rz(d01);
        const float u10 = hgb::f64_to_f32_rz(d10), u11 = hgb::f64_to_f32_rz(d11);
        int sent = 0;
        float above = 0.0f;
        {
            const long long bb[4] = {b00, b01, b10, b11};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const bool is = bb[c] == hgb::F64_MINUS_ONE_BITS;
                sent += is;
                bad |= bb[c] < 0 && !is && bb[c] != (long long)0x8000000000000000ull &&
                       (unsigned long long)bb[c] <= 0xFFF0000000000000ull;   // < 0, not -1, -0, NaN
            }
            if (sent == 0)
                above = (hgb::f64_to_f32_rz(__longlong_as_double(b10)) + hgb::f64_to_f32_rz(__longlong_as_double(b00))) +
                        (hgb::f64_to_f32_rz(__longlong_as_double(b11)) + hgb::f64_to_f32_rz(__longlong_as_double(b01)));
        }
        if (z > z0) {   // vertex z closes bin z - 1
            const long out = ((long)cell * nzb + (z - 1)) * g.nf + f;
            // number: Kahan sum of the eight vertices (sam_cyutils.pyx:199-214)
            hgb::Kahan32 acc;
            acc.add(n00);
            acc.add(u00);
            acc.add(n01);
            acc.add(u01);
            acc.add(n10);
            acc.add(u10);
            acc.add(n11);
            acc.add(u11);
            number[out] = hgb::f32_to_f64_scaled(acc.s * s_vol[z - 1] * dlnf, 0);
            // strain (gravwaves.py:694-724)
            const int n_sent = below_sent + sent;
            float zb = 0.0f;
            if (n_sent == 0) {   // all corners >= 0: the midpoints cannot cancel
                zb = 0.125f * (above + below);
            } else if (n_sent < 8) {   // the sentinel enters the mean: the reference's FP64 midpoints
                const double a00 = 0.5 * (__longlong_as_double(l10) + __longlong_as_double(l00));
                const double a01 = 0.5 * (__longlong_as_double(b10) + __longlong_as_double(b00));
                const double a10 = 0.5 * (__longlong_as_double(l11) + __longlong_as_double(l01));
                const double a11 = 0.5 * (__longlong_as_double(b11) + __longlong_as_double(b01));
                const double zd = 0.5 * (0.5 * (a11 + a01) + 0.5 * (a10 + a00));
                zb = (zd > 0.0) ? hgb::f64_to_f32_rz(zd) : 0.0f;
            }
            double res = 0.0;
            if (zb > 0.0f) {
                const float dc = dc_over_dh_f32(s, zb);
                const float zp1 = 1.0f + zb;
                const float zp23 = zp1 * rcbrtf(zp1);
                const float hs = __fdividef(amp_mq * amp_f * zp23, dc);
                res = hgb::f32_to_f64_scaled(hs * hs * fcdf, e2);
            }
            h2fdf[out] = res;
        }
        n00 = u00; n01 = u01; n10 = u10; n11 = u11;
        l00 = b00; l01 = b01; l10 = b10; l11 = b11;
        below = above;
        below_sent = sent;
    }
    if (bad) hgb::flag(d_status, HGB_STATUS_INVALID_REDSHIFT);
}

// single_sources.py:117-143 on one (bin, frequency): the redshift midpoints (same order as
// k_cells), -1 where not positive; comoving distance (+inf there); Kepler separation at the
// rest-frame orbital frequency; angular separation.  IEEE semantics give the reference's inf / NaN
// for the -1 bins.  Also records the largest finite magnitude of each grid (as a frexp exponent)
// over the bins with nonzero strain.
// FP64 bounds it, the power above all, so bins without a redshift (two thirds, in runs along the
// frequencies) take none: their separation is infinite.  The exponents are read off the bits and go to
// memory once a block, if at all.  40x30x36 bins, 20 frequencies: 303 us before, 237 us now.
constexpr int PG_THREADS = 256;

// frexp's exponent of a finite nonzero number, INT_MIN of any other
__device__ __forceinline__ int binary_exponent(double x) {
    const long long b = __double_as_longlong(x);
    const int field = (int)(b >> 52) & 0x7FF;
    if (field == 0x7FF || (b << 1) == 0) return INT_MIN;
    if (field == 0) {
        int e;
        frexp(x, &e);
        return e;
    }
    return field - 1022;
}

__global__ void __launch_bounds__(PG_THREADS) k_param_grids(BinGeom g, const double *__restrict__ mt_cent, const double *__restrict__ fobs_cent,
                              const double *__restrict__ redz_final, double nwtg, StrainArgs s,
                              const double *__restrict__ h2fdf, double *__restrict__ rz_mid,
                              double *__restrict__ dcom, double *__restrict__ sepa, double *__restrict__ angs,
                              int *scale_log2) {
    const long nb = (long)(g.nm - 1) * (g.nq - 1) * (g.nz - 1);
    const long idx = (long)blockIdx.x * PG_THREADS + threadIdx.x;
    __shared__ int s_e[4];
    if (threadIdx.x < 4) s_e[threadIdx.x] = INT_MIN;
    __syncthreads();
    int e[4] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN};
    if (idx < nb * g.nf) {
        const int f = (int)(idx % g.nf);
        const long b = idx / g.nf;
        const int z = (int)(b % (g.nz - 1));
        const int q = (int)((b / (g.nz - 1)) % (g.nq - 1));
        const int m = (int)(b / ((long)(g.nz - 1) * (g.nq - 1)));
        double r[2][2][2];
#pragma unroll
        for (int ii = 0; ii < 2; ii++)
#pragma unroll
            for (int jj = 0; jj < 2; jj++)
#pragma unroll
                for (int kk = 0; kk < 2; kk++) r[ii][jj][kk] = redz_final[vtx(g, m + ii, q + jj, z + kk, f)];
        const double a00 = 0.5 * (r[1][0][0] + r[0][0][0]);
        const double a01 = 0.5 * (r[1][0][1] + r[0][0][1]);
        const double a10 = 0.5 * (r[1][1][0] + r[0][1][0]);
        const double a11 = 0.5 * (r[1][1][1] + r[0][1][1]);
        const double b0 = 0.5 * (a10 + a00);
        const double b1 = 0.5 * (a11 + a01);
        double zb = 0.5 * (b1 + b0);
        double dc = INFINITY;
        if (zb > 0.0) dc = hgb::comoving_distance(s.dc_val, s.dc_der, s.dc_n, zb);
        else zb = -1.0;
        const double frst = fobs_cent[f] * (1.0 + zb);
        const double w = 2.0 * HGB_PI * frst;
        const double arg = nwtg * mt_cent[m] / (w * w);
        const double sp = arg == INFINITY ? arg : pow(arg, 1.0 / 3.0);
        const double an = sp / (dc / (1.0 + zb));
        rz_mid[idx] = zb;
        dcom[idx] = dc;
        sepa[idx] = sp;
        angs[idx] = an;
        if (scale_log2 && (!h2fdf || h2fdf[idx] != 0.0)) {
            e[0] = binary_exponent(zb);
            e[1] = binary_exponent(dc);
            e[2] = binary_exponent(sp);
            e[3] = binary_exponent(an);
        }
    }
    if (!scale_log2) return;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int top = __reduce_max_sync(0xffffffffu, e[k]);
        if ((threadIdx.x & 31) == 0 && top != INT_MIN) atomicMax(s_e + k, top);
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_e[threadIdx.x] > *(volatile int *)(scale_log2 + threadIdx.x))
        atomicMax(scale_log2 + threadIdx.x, s_e[threadIdx.x]);
}

}  // namespace

extern "C" {

int hgb_param_grids(const double *mt_cent, int n_mtot, int n_mrat, int n_redz, const double *fobs_orb_cent,
                    int n_freq, const double *redz_final, double nwtg, const hgb_cosmo *cosmo,
                    const double *h2fdf, double *redz_mid, double *dcom, double *sepa, double *angs,
                    int *scale_log2, void *stream) {
    HGB_CHECK_ARG(mt_cent && fobs_orb_cent && redz_final && cosmo && redz_mid && dcom && sepa && angs);
    HGB_CHECK_ARG(n_mtot >= 2 && n_mrat >= 2 && n_redz >= 2 && n_freq >= 1);
    HGB_CHECK_ARG(cosmo->dc_val && cosmo->dc_der && cosmo->dc_n >= 2);
    BinGeom g{n_mtot, n_mrat, n_redz, n_freq};
    const StrainArgs s = strain_args(0.0, cosmo);
    cudaStream_t st = (cudaStream_t)stream;
    if (scale_log2) {
        cudaError_t err = cudaMemsetAsync(scale_log2, 0x80, 4 * sizeof(int), st);   // very negative
        if (err != cudaSuccess) {
            hgb::set_cuda_error(err);
            return HGB_ERR_CUDA;
        }
    }
    const long n = (long)(n_mtot - 1) * (n_mrat - 1) * (n_redz - 1) * n_freq;
    k_param_grids<<<(unsigned)hgb::ceil_div(n, PG_THREADS), PG_THREADS, 0, st>>>(g, mt_cent, fobs_orb_cent, redz_final, nwtg, s,
                                                                   h2fdf, redz_mid, dcom, sepa, angs, scale_log2);
    return hgb::check_launch();
}

int hgb_integrate_3dx1d(const double *log10_mtot, int n_mtot, const double *mrat, int n_mrat, const double *redz,
                        int n_redz, const double *dln_freq, int n_freq, const double *dnum, double *number,
                        void *stream) {
    HGB_CHECK_ARG(log10_mtot && mrat && redz && dln_freq && dnum && number);
    HGB_CHECK_ARG(n_mtot >= 2 && n_mrat >= 2 && n_redz >= 2 && n_freq >= 1);
    BinGeom g{n_mtot, n_mrat, n_redz, n_freq};
    const StrainArgs s{0.0, nullptr, nullptr, nullptr, 0, -1, 0.0};
    const long cells = (long)(n_mtot - 1) * (n_mrat - 1);
    const CellSplit sp = cell_split(n_freq, n_redz - 1, cells, CELL_THREADS);
    const dim3 grid((unsigned)cells, (unsigned)sp.parts);
    k_cells<true, false><<<grid, sp.threads, 0, (cudaStream_t)stream>>>(g, sp, s, nullptr, log10_mtot, mrat, redz, nullptr,
                                                                  dln_freq, dnum, nullptr, number, nullptr, nullptr);
    return hgb::check_launch();
}

int hgb_char_strain_sq(const double *mtot, int n_mtot, const double *mrat, int n_mrat, int n_redz,
                       const double *fobs_orb_edges, int n_freq, const double *redz_final, double gw_src_const,
                       const hgb_cosmo *cosmo, double *h2fdf, int *d_status, void *stream) {
    HGB_CHECK_ARG(mtot && mrat && fobs_orb_edges && redz_final && cosmo && h2fdf);
    HGB_CHECK_ARG(n_mtot >= 2 && n_mrat >= 2 && n_redz >= 2 && n_freq >= 1);
    HGB_CHECK_ARG(cosmo->dc_val && cosmo->dc_der && cosmo->dc_n >= 2);
    BinGeom g{n_mtot, n_mrat, n_redz, n_freq};
    HGB_CHECK_ARG(n_freq <= STRAIN_MAX_FREQ);
    const StrainArgs s = strain_args(gw_src_const, cosmo);
    const long cells = (long)(n_mtot - 1) * (n_mrat - 1);
    const CellSplit sp = cell_split(n_freq, n_redz - 1, cells, CELL_THREADS);
    const dim3 grid((unsigned)cells, (unsigned)sp.parts);
    k_cells<false, true><<<grid, sp.threads, 0, (cudaStream_t)stream>>>(g, sp, s, mtot, nullptr, mrat, nullptr, fobs_orb_edges,
                                                                     nullptr, nullptr, redz_final, nullptr, h2fdf,
                                                                     d_status);
    return hgb::check_launch();
}

int hgb_number_and_strain_f32(const double *mtot, const double *log10_mtot, int n_mtot, const double *mrat,
                              int n_mrat, const double *redz, int n_redz, const double *fobs_orb_edges,
                              const double *dln_freq, int n_freq, const double *dnum, const double *redz_final,
                              double gw_src_const, const hgb_cosmo *cosmo, double *number, double *h2fdf,
                              int *d_status, void *stream) {
    HGB_CHECK_ARG(mtot && log10_mtot && mrat && redz && fobs_orb_edges && dln_freq && dnum && redz_final);
    HGB_CHECK_ARG(cosmo && number && h2fdf);
    HGB_CHECK_ARG(n_mtot >= 2 && n_mrat >= 2 && n_redz >= 2 && n_freq >= 1 && n_freq <= F32_MAX_FREQ);
    HGB_CHECK_ARG(cosmo->dcg_val && cosmo->dcg_der && cosmo->dc_n >= 2 && cosmo->hubble_distance > 0.0);
    HGB_CHECK_ARG(gw_src_const > 0.0);
    BinGeom g{n_mtot, n_mrat, n_redz, n_freq};
    StrainArgs32 s{cosmo->dcg_val, cosmo->dcg_der, cosmo->dc_n, 1.0f / (float)cosmo->dc_n};
    const long cells = (long)(n_mtot - 1) * (n_mrat - 1);
    const CellSplit sp = cell_split(n_freq, n_redz - 1, cells, CELL_F32_THREADS);
    const dim3 grid((unsigned)cells, (unsigned)sp.parts);
    size_t smem = sizeof(float) * (size_t)(n_redz - 1);
    HGB_CHECK_ARG(smem <= 32 * 1024);
    k_cells_f32<<<grid, sp.threads, smem, (cudaStream_t)stream>>>(g, sp, s, gw_src_const / cosmo->hubble_distance, mtot,
                                                             log10_mtot, mrat, redz, fobs_orb_edges, dln_freq, dnum,
                                                             redz_final, number, h2fdf, d_status);
    return hgb::check_launch();
}

int hgb_number_and_strain(const double *mtot, const double *log10_mtot, int n_mtot, const double *mrat, int n_mrat,
                          const double *redz, int n_redz, const double *fobs_orb_edges, const double *dln_freq,
                          int n_freq, const double *dnum, const double *redz_final, double gw_src_const,
                          const hgb_cosmo *cosmo, double *number, double *h2fdf, int *d_status, void *stream) {
    HGB_CHECK_ARG(mtot && log10_mtot && mrat && redz && fobs_orb_edges && dln_freq && dnum && redz_final);
    HGB_CHECK_ARG(cosmo && number && h2fdf);
    HGB_CHECK_ARG(n_mtot >= 2 && n_mrat >= 2 && n_redz >= 2 && n_freq >= 1);
    HGB_CHECK_ARG(cosmo->dc_val && cosmo->dc_der && cosmo->dc_n >= 2);
    BinGeom g{n_mtot, n_mrat, n_redz, n_freq};
    HGB_CHECK_ARG(n_freq <= STRAIN_MAX_FREQ);
    const StrainArgs s = strain_args(gw_src_const, cosmo);
    const long cells = (long)(n_mtot - 1) * (n_mrat - 1);
    const CellSplit sp = cell_split(n_freq, n_redz - 1, cells, CELL_THREADS);
    const dim3 grid((unsigned)cells, (unsigned)sp.parts);
    k_cells<true, true><<<grid, sp.threads, 0, (cudaStream_t)stream>>>(g, sp, s, mtot, log10_mtot, mrat, redz, fobs_orb_edges,
                                                                    dln_freq, dnum, redz_final, number, h2fdf, d_status);
    return hgb::check_launch();
}

}  // extern "C"
