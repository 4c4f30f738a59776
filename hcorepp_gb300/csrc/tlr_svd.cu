// Core of the recompression: M = R_U R_V^T, its SVD by one-sided Jacobi, the rank
// truncation, and the new left/right factors in the small basis.
//
// Replaces the R extraction + core GEMM + SVD + CalculateNewRank + CalculateVTnew of
// CompressedTile<T>::Gemm (src/operators/concrete/Compressed.cpp:441-527, :597-599) and the
// host-synchronising rank scan of the CUDA backend (src/kernels/cuda/CudaKernels.cu:656-697).
//
// One team per update: a quarter or half of a CTA, or a cluster of CTAs for a core that does not fit half the
// shared memory.  M = R_U R_V^T on DMMA; Householder QR with column pivoting of M,
// stopped once the remaining columns lie far below the truncation threshold; one-sided Jacobi on
// the rk columns of X = R^T until every pair is orthogonal to working precision: X J = W,
// sigma_j = ||w_j||, found in single precision and finished in FP64 (jacobi_precond; small cores by FP64 sweeps
// alone).  The right factor is XV = P W_r (= V_r Sigma_r) and the left one U = M XV Sigma^-2 (= U_r).
// The pivoted QR runs in FP64 (plain form, wide cores) or float-float (mixed form).  The rank rule is the
// reference's (omp/kernels.cpp:82-104) applied to the sorted sigma.
//
// Measured (1.06 TFLOP/s FP64 pipe): the sweeps of a 200-column core of stack width 215 took 72,500 kcycles
// on one SM, 4,970 on its cluster of eight; of a 25-column core 930, now 348, four to an SM; the pivoted QR
// 9,970 -> 2,140 and 274 -> 236.
#include <algorithm>
#include <cfloat>

#include "internal.cuh"
#include "df.cuh"

namespace hcgb {

namespace {

constexpr int SVD_THREADS = 512;
constexpr int WIDE_POOL_DOUBLES = 16640;  // shared memory of a CTA: 130 KB leave the rest to L1 ...
constexpr int WIDE_POOL_K = 350;          // ... up to the width whose columns they hold
constexpr float PRECOND_TOL32 = 1e-6f;  // above the rounding of a single-precision cosine
constexpr int PRECOND_MAX_SWEEPS = 12;
constexpr int SVD_RED_DOUBLES = 64, SVD_REDI_INTS = 128;  // reduction area (up to 32 warps)
constexpr int SVD_AUX_FIXED = 1 + SVD_RED_DOUBLES + SVD_REDI_INTS / 2;  // aux = 6 kmax + this

__device__ __forceinline__ void jacobi_pair(int t, int pp, int n2, int &i, int &j) {
    const int nm1 = n2 - 1;
    if (pp == 0) {
        i = 0;
        j = 1 + t % nm1;
    } else {
        i = 1 + (pp + t) % nm1;
        j = 1 + (n2 - 1 - pp + t) % nm1;
    }
}

template <typename T>
__device__ __forceinline__ T group_sum(T v, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <>
__device__ __forceinline__ df group_sum<df>(df v, int G) {
    return df_group_sum(v, G);
}

// Tangent of the Jacobi angle that orthogonalises a pair with squared norms a, b and inner
// product c: zeta = (b - a) / (2 c), t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)) (Rutishauser).
// Evaluated in single precision after scaling both terms by the same power of two (read off the
// exponent of c with integer operations), so no double-precision divide or square root is spent
// on it; the rotation built from t is orthogonal to working precision whatever t's rounding.
__device__ __forceinline__ float jacobi_tangent(double a, double b, double c) {
    const int hi = __double2hiint(c);
    const int e = ((hi >> 20) & 0x7ff) - 1023;
    const int se = e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
    const double scale = __hiloint2double((1023 - se) << 20, 0);  // 2^-se, exact
    const float num = (float) ((b - a) * scale);
    const float den = (float) (2.0 * c * scale);
    const float zf = num / den;
    if (fabsf(zf) > 1.0e18f) return 0.5f / zf;
    return copysignf(1.0f, zf) / (fabsf(zf) + sqrtf(fmaf(zf, zf, 1.0f)));
}

// A rotated pair's bookkeeping (tracked squared norms a - t cd, b + t cd; scales d cos; inverse scales
// (1/d) q cos) spread over the first four lanes of its group: every lane evaluates the same three FP64
// instructions on operands it selects, instead of one lane issuing six or seven (the FP64 pipe, one
// warp-wide instruction per ~19 cycles per SM on GB300, bounds the plain core).  Lanes 0 / 1 store
// column i's / j's norm and inverse scale, lanes 2 / 3 its scale.
__device__ __forceinline__ void pair_bookkeeping(int gl, int i, int j, double a, double b, double tt, double cd,
                                                 double cs, double q, double di, double dj, double dvi, double dvj,
                                                 double *nrm, double *dsc, int dstride) {
    const bool second = gl & 1, norm_lane = gl < 2;
    const int col = second ? j : i;
    const double m1 = norm_lane ? (second ? tt : -tt) : (second ? dj : di);
    const double v = fma(m1, norm_lane ? cd : cs, norm_lane ? (second ? b : a) : 0.0);
    const double w = (second ? dvj : dvi) * (q * cs);
    if (norm_lane) {
        nrm[col] = v;
        dsc[dstride + col] = w;
    } else if (gl < 4) {
        dsc[col] = v;
    }
}

// One sweep of one-sided Jacobi over the `ncols` columns (length `rows`) of X (ld ldx), with G
// lanes per column pair (32/G pairs per warp at a time) and up to RPL rows per lane in registers.
// Squared column norms are tracked in nrm[] (a' = a - t c, b' = b + t c), so each pair costs one
// inner product.  A pair is rotated when c^2 > tol2 a b and both columns are above the noise
// floor `tiny`; columns below it hold only rounding errors of the larger ones.
//
// The rotations are applied in scaled form (the idea of fast Givens rotations): column i is
// stored as x_i with the true column d_i x_i, so the rotation
//   X_i' = cos (X_i - t X_j),  X_j' = cos (X_j + t X_i)
// becomes x_i' = x_i - t (d_j / d_i) x_j, x_j' = x_j + t (d_i / d_j) x_i, d' = cos d: one FMA per
// element instead of a multiply and an FMA.  d and 1/d live in dsc[0..) and dsc[dstride..);
// the caller folds them back into the columns at the start of every sweep.
template <int G, int RPL, class TM>
__device__ int jacobi_sweep(const TM &tm, double *X, int ldx, int rows, int ncols, double *nrm, double tol2,
                            double tiny, int n2, double *dsc, int dstride) {
    static_assert(G >= 4, "pair_bookkeeping spreads a pair's bookkeeping over four lanes");
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int PPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    const int npairs = n2 / 2;
    const int nchunks = (npairs + PPW - 1) / PPW;
    int rotations = 0;
    for (int t = 0; t < n2 - 1; t++) {
        for (int ch = warp; ch < nchunks; ch += nw) {
            const int pp = ch * PPW + grp;
            int i = 0, j = 0;
            bool act = pp < npairs;
            if (act) {
                jacobi_pair(t, pp, n2, i, j);
                act = i < ncols && j < ncols;
            }
            double *x = X + (size_t) (act ? i : 0) * ldx;
            double *y = X + (size_t) (act ? j : 0) * ldx;
            double xr[RPL], yr[RPL];
            double c = 0.0;
#pragma unroll
            for (int q = 0; q < RPL; q++) {
                xr[q] = yr[q] = 0.0;
                if (G * q < rows) {  // uniform across the warp: whole row slots beyond `rows` are skipped
                    const int r = gl + G * q;
                    if (act && r < rows) {
                        xr[q] = x[r];
                        yr[q] = y[r];
                    }
                    c = fma(xr[q], yr[q], c);
                }
            }
            c = group_sum(c, G);
            const double a = act ? nrm[i] : 0.0, b = act ? nrm[j] : 0.0;
            double di = 1.0, dj = 1.0;
            if (act) {
                di = dsc[i];
                dj = dsc[j];
            }
            const double cd = c * di * dj;  // true inner product
            const bool rot = act && a > tiny && b > tiny && cd * cd > tol2 * a * b;
            if (rot) {
                const double tt = (double) jacobi_tangent(a, b, cd);
                const double q = fma(tt, tt, 1.0);
                const double cs = rsqrt(q);
                const double dvi = dsc[dstride + i], dvj = dsc[dstride + j];
                const double t1 = tt * dj * dvi, t2 = tt * di * dvj;
#pragma unroll
                for (int q2 = 0; q2 < RPL; q2++) {
                    if (G * q2 < rows) {
                        const int r = gl + G * q2;
                        if (r < rows) {
                            x[r] = fma(-t1, yr[q2], xr[q2]);
                            y[r] = fma(t2, xr[q2], yr[q2]);
                        }
                    }
                }
                pair_bookkeeping(gl, i, j, a, b, tt, cd, cs, q, di, dj, dvi, dvj, nrm, dsc, dstride);
                if (gl == 0) rotations++;
            }
        }
        tm.sync();
    }
    return rotations;
}

// The same sweep with the column pairs read from memory by G-lane groups in a loop over the rows
// instead of register tiles (rows of any length, 32 / G pairs per warp): for long columns it packs
// more pairs into each warp instruction than the register tiles can, which shares the per-pair
// scalar FP64 work among more pairs at the price of reading the columns twice.
template <int G, class TM>
__device__ int jacobi_sweep_loop(const TM &tm, double *X, int ldx, int rows, int ncols, double *nrm, double tol2,
                                 double tiny, int n2, double *dsc, int dstride) {
    static_assert(G >= 4, "pair_bookkeeping spreads a pair's bookkeeping over four lanes");
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int PPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    const int npairs = n2 / 2;
    const int nchunks = (npairs + PPW - 1) / PPW;
    int rotations = 0;
    for (int t = 0; t < n2 - 1; t++) {
        for (int ch = warp; ch < nchunks; ch += nw) {
            const int pp = ch * PPW + grp;
            int i = 0, j = 0;
            bool act = pp < npairs;
            if (act) {
                jacobi_pair(t, pp, n2, i, j);
                act = i < ncols && j < ncols;
            }
            double *x = X + (size_t) (act ? i : 0) * ldx;
            double *y = X + (size_t) (act ? j : 0) * ldx;
            double c0 = 0.0, c1 = 0.0;
            if (act) {
                int r = gl;
                for (; r + G < rows; r += 2 * G) {
                    c0 = fma(x[r], y[r], c0);
                    c1 = fma(x[r + G], y[r + G], c1);
                }
                if (r < rows) c0 = fma(x[r], y[r], c0);
            }
            const double c = group_sum(c0 + c1, G);
            const double a = act ? nrm[i] : 0.0, b = act ? nrm[j] : 0.0;
            double di = 1.0, dj = 1.0;
            if (act) {
                di = dsc[i];
                dj = dsc[j];
            }
            const double cd = c * di * dj;  // true inner product
            const bool rot = act && a > tiny && b > tiny && cd * cd > tol2 * a * b;
            if (rot) {
                const double tt = (double) jacobi_tangent(a, b, cd);
                const double q = fma(tt, tt, 1.0);
                const double cs = rsqrt(q);
                const double dvi = dsc[dstride + i], dvj = dsc[dstride + j];
                const double t1 = tt * dj * dvi, t2 = tt * di * dvj;
#pragma unroll 4
                for (int r = gl; r < rows; r += G) {
                    const double xv = x[r], yv = y[r];
                    x[r] = fma(-t1, yv, xv);
                    y[r] = fma(t2, xv, yv);
                }
                pair_bookkeeping(gl, i, j, a, b, tt, cd, cs, q, di, dj, dvi, dvj, nrm, dsc, dstride);
                if (gl == 0) rotations++;
            }
        }
        tm.sync();
    }
    return rotations;
}

// Jacobi iteration on X: exact squared column norms at the start of every sweep (the scales of
// the previous sweep folded into the columns), then sweeps until no pair rotates (or max_sweeps).
// RPL = 0 selects the looped sweep.
template <int G, int RPL, class TM>
__device__ void jacobi(const TM &tm, double *X, int ldx, int rows, int ncols, double *nrm, int *s_rot,
                       double *s_amax, int *sweeps_out, bool *converged_out, double tol, int max_sweeps, double *dsc,
                       int dstride) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    const double tol2 = tol * tol;
    const double noise = DBL_EPSILON * (double) (rows > 1 ? rows : 1);
    const int n2 = ncols + (ncols & 1);
    int sweeps = 0;
    bool converged = ncols < 2;
    for (int j = tm.tid; j < ncols; j += tm.nth) dsc[j] = dsc[dstride + j] = 1.0;
    tm.sync();
    auto fold_and_norms = [&](double &amax) {
        for (int j = warp; j < ncols; j += nw) {
            double *col = X + (size_t) j * ldx;
            const double dj = dsc[j];
            double sq = 0.0;
            for (int r = lane; r < rows; r += 32) {
                double v = col[r];
                if (dj != 1.0) {
                    v *= dj;
                    col[r] = v;
                }
                sq = fma(v, v, sq);
            }
            sq = warp_sum(sq);
            if (lane == 0) {
                nrm[j] = sq;
                dsc[j] = dsc[dstride + j] = 1.0;
            }
            amax = fmax(amax, sq);
        }
    };
    while (!converged && sweeps < max_sweeps) {
        if (tm.tid == 0) {
            *s_rot = 0;
            *s_amax = 0.0;
        }
        tm.sync();
        double amax = 0.0;
        fold_and_norms(amax);
        if (lane == 0) atomicMax(reinterpret_cast<unsigned long long *>(s_amax), __double_as_longlong(amax));
        tm.sync();
        const double tiny = *s_amax * noise * noise;
        int rot;
        if constexpr (RPL == 0)
            rot = jacobi_sweep_loop<G>(tm, X, ldx, rows, ncols, nrm, tol2, tiny, n2, dsc, dstride);
        else
            rot = jacobi_sweep<G, RPL>(tm, X, ldx, rows, ncols, nrm, tol2, tiny, n2, dsc, dstride);
        if (rot) atomicAdd(s_rot, rot);
        tm.sync();
        sweeps++;
        converged = (*s_rot == 0);
        tm.sync();
    }
    double amax = 0.0;
    fold_and_norms(amax);  // a sweep limit can leave scales unfolded
    tm.sync();
    *sweeps_out = sweeps;
    *converged_out = converged;
}

// Lane-group / register-tile choice for a column length: G lanes per pair, RPL rows per lane.
template <int MAXRPL, class TM>
__device__ void jacobi_dispatch(const TM &tm, double *X, int ldx, int rows, int ncols, double *nrm, int *s_rot,
                                double *s_amax, int *sweeps, bool *conv, double tol, int max_sweeps, double *dsc,
                                int dstride, bool x_in_smem) {
    // Fewer lanes per pair put more pairs in one warp instruction, so the per-pair scalar work
    // (tangent, tests, norm updates), which runs as full-width FP64 warp instructions on a pipe that
    // issues one of them per ~19 cycles per SM, is shared by 4-8 pairs; RPL rows per lane stay in
    // registers.  (Two lanes per pair for columns of up to 32 rows, one warp taking every pair of a
    // step, measured slower: 760 vs 673 kcycles per 17-32-column core.)
    // Longer columns held in shared memory: 4- or 8-lane groups in a loop over the rows (8 or 4 pairs
    // per warp instruction; each pair is read twice).  Columns in the workspace (cores too wide for
    // the team's shared memory) keep register tiles, which read them once: the loop measured 15-35 %
    // slower there (long-scoreboard stalls on the second read).
    if (rows <= 32) jacobi<4, 8>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 64 && MAXRPL >= 16) jacobi<4, 16>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 64) jacobi<8, 8>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (x_in_smem && rows <= 128) jacobi<4, 0>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (x_in_smem) jacobi<8, 0>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 128 && MAXRPL >= 16) jacobi<8, 16>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 128) jacobi<16, 8>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 256 && MAXRPL >= 16) jacobi<16, 16>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    else if (rows <= 256) jacobi<32, 8>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
    // Longer columns (nb = 1024 stacks): the register tile that would cover them spills, so the loop.
    else jacobi<8, 0>(tm, X, ldx, rows, ncols, nrm, s_rot, s_amax, sweeps, conv, tol, max_sweeps, dsc, dstride);
}

// ---------------------------------------------------------------------------------------------
// Preconditioning of the FP64 Jacobi.  One FP64 warp instruction takes ~19 cycles of an SM here, an FP32
// one a quarter of a cycle, so the sweeps that only have to find the rotations run in single precision:
//   1. one-sided Jacobi on X32 = X 2^-e with the rotations accumulated in J32 (jacobi32_sweep);
//   2. J = J32 (I + H), H = -E/2 + 3/8 E^2 - 5/16 E^3, E = J32^T J32 - I: the orthogonal polar factor of
//      J32 (Newton-Schulz series; E is formed from exact products, so J is orthogonal to ~1e-15);
//   3. W = X J in FP64: orthogonal columns up to cosines of ~1e-6;
//   4. corrections W <- W exp(S) (jacobi_correct): S holds every pair's rotation angle, the cosines come
//      from a float-float Gram matrix and W S is added to W in FP64.  The angles are small, so the rotations
//      of all pairs commute up to second order and two corrections reach working precision.
// Only step 3 and one addition per element and correction use the FP64 pipe.  A pair that would turn
// by more than CORRECT_MAX_TAN (nearly equal singular values), or a correction that does not converge,
// leaves the rest to the FP64 sweeps.
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Tangent of the rotation angle, zeta = (b - a) / (2 c) (Rutishauser; zeta^2 must not overflow).
__device__ __forceinline__ float rotation_tangent(float zeta) {
    if (fabsf(zeta) > 1.0e18f) return 0.5f / zeta;
    return copysignf(1.f, zeta) / (fabsf(zeta) + sqrtf(fmaf(zeta, zeta, 1.f)));
}

// Cosine and sine of the single-precision sweeps.  The chain of two divisions and two square roots was half of a
// step's latency; approximations do (any tangent gives a rotation), but the cosine gets a Newton step: its
// error makes the accumulated J32 less orthogonal.
__device__ __forceinline__ void rotation32(float a, float b, float c, float &cs, float &sn) {
    const float zeta = __fdividef(b - a, 2.f * c), z = fabsf(zeta);
    float t = z > 1.0e18f ? __fdividef(0.5f, z) : __fdividef(1.f, z + sqrt_approx(fmaf(z, z, 1.f)));
    t = copysignf(t, zeta);
    const float q = fmaf(t, t, 1.f), r = rsqrtf(q);
    cs = fmaf(0.5f * r, fmaf(-q * r, r, 1.f), r);
    sn = cs * t;
}

// Pair `pp` of step t over columns [0, nc_a) and [off_b, off_b + nc_b): round robin over all of them (cross =
// false) or one column of each range.  Returns whether the step has such a pair.
__device__ __forceinline__ bool sweep_pair(int t, int pp, int nc_a, int nc_b, int off_b, bool cross, int &i, int &j) {
    if (cross) {
        const int wide = nc_a > nc_b ? nc_a : nc_b;
        const int q = pp + t < wide ? pp + t : pp + t - wide;
        i = pp;
        j = off_b + q;
        return t < wide && pp < nc_a && q < nc_b;
    }
    const int nc = nc_a + nc_b, n2 = nc + (nc & 1);
    if (t >= n2 - 1 || pp >= n2 / 2) return false;
    jacobi_pair(t, pp, n2, i, j);
    if (i >= nc || j >= nc) return false;
    i = i < nc_a ? i : off_b + i - nc_a;
    j = j < nc_a ? j : off_b + j - nc_a;
    return true;
}

// Rotates columns x and y (x4 quads of X32, then j4 of J32, zero padded) by G lanes when their cosine exceeds tol;
// the inner products take the first part, the rotation both.  Every lane of the warp calls.
template <int G>
__device__ __forceinline__ int jacobi32_rotate(bool act, float4 *x, float4 *y, int x4, int j4, int gl, float tol) {
    float a = 0.f, b = 0.f, c = 0.f;
    if (act) {
#pragma unroll 4
        for (int r = gl; r < x4; r += G) {
            const float4 u = x[r], v = y[r];
            a = fmaf(u.x, u.x, fmaf(u.y, u.y, fmaf(u.z, u.z, fmaf(u.w, u.w, a))));
            b = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, b))));
            c = fmaf(u.x, v.x, fmaf(u.y, v.y, fmaf(u.z, v.z, fmaf(u.w, v.w, c))));
        }
    }
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (!(act && a > 0.f && b > 0.f && fabsf(c) * rsqrtf(a) * rsqrtf(b) > tol)) return 0;
    float cs, sn;
    rotation32(a, b, c, cs, sn);
#pragma unroll 4
    for (int r = gl; r < x4 + j4; r += G) {
        const float4 u = x[r], v = y[r];
        x[r] = make_float4(fmaf(cs, u.x, -sn * v.x), fmaf(cs, u.y, -sn * v.y), fmaf(cs, u.z, -sn * v.z),
                           fmaf(cs, u.w, -sn * v.w));
        y[r] = make_float4(fmaf(cs, v.x, sn * u.x), fmaf(cs, v.y, sn * u.y), fmaf(cs, v.z, sn * u.z),
                           fmaf(cs, v.w, sn * u.w));
    }
    return gl == 0;
}

// One sweep over the columns of Y (ls4 quads apart), in shared memory: round robin (blocks = 0), or the cluster's
// order of column blocks (blocks = their number: jacobi32_blocks), block pairs side by side, so that a core gives the
// same result on one SM and on a cluster.
template <int G, class TM>
__device__ int jacobi32_sweep(const TM &tm, float4 *Y, int ls4, int x4, int j4, int nc, int blocks, float tol) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int PPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    const int w = blocks ? (nc + blocks - 1) / blocks : nc, per = blocks ? w : (nc + 1) / 2;
    const int npairs = blocks ? blocks / 2 * per : per, nchunks = (npairs + PPW - 1) / PPW;
    const int rounds = blocks ? blocks - 1 : 1, n2 = nc + (nc & 1);
    int rotations = 0;
    for (int round = 0; round < rounds; round++) {
        const int steps = blocks ? (round ? w : 2 * w - 1) : n2 - 1;
        for (int t = 0; t < steps; t++) {
            for (int ch = warp; ch < nchunks; ch += nw) {
                const int id = ch * PPW + grp;
                int i = 0, j = 0;
                bool act = id < npairs;
                if (act && blocks) {
                    int bi, bj;
                    jacobi_pair(round, id / per, blocks, bi, bj);
                    const int ra = nc - bi * w, rb = nc - bj * w;
                    const int na = ra < 0 ? 0 : (ra < w ? ra : w), nb = rb < 0 ? 0 : (rb < w ? rb : w);
                    act = sweep_pair(t, id % per, na, nb, (bj - bi) * w, round > 0, i, j);
                    i += bi * w;
                    j += bi * w;
                } else if (act) {
                    act = sweep_pair(t, id, nc, 0, 0, false, i, j);
                }
                rotations += jacobi32_rotate<G>(act, Y + (size_t) (act ? i : 0) * ls4, Y + (size_t) (act ? j : 0) * ls4, x4,
                                                j4, gl, tol);
            }
            tm.sync();
        }
    }
    return rotations;
}

// The steps of one block pair (columns [0, nc_a) and [off_b, off_b + nc_b) of Y, ls4 quads apart) by one CTA.
template <int G, class TM>
__device__ int jacobi32_block_pair(const TM &tm, float4 *Y, int ls4, int x4, int j4, int nc_a, int nc_b, int off_b,
                                   bool cross, float tol) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int PPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    const int nc = nc_a + nc_b, n2 = nc + (nc & 1), wide = nc_a > nc_b ? nc_a : nc_b;
    const int npairs = cross ? wide : n2 / 2, steps = cross ? wide : n2 - 1;
    int rotations = 0;
    for (int t = 0; t < steps; t++) {
        for (int p0 = warp * PPW; p0 < npairs; p0 += nw * PPW) {
            int i = 0, j = 0;
            const bool act = sweep_pair(t, p0 + grp, nc_a, nc_b, off_b, cross, i, j);
            rotations += jacobi32_rotate<G>(act, Y + (size_t) (act ? i : 0) * ls4, Y + (size_t) (act ? j : 0) * ls4, x4, j4,
                                            gl, tol);
        }
        tm.sync();
    }
    return rotations;
}

// 8 R x 4 R output tiles of an M x N result, one warp each: lane (li, lj) accumulates rows i0 + li + 8 u and columns
// j0 + lj + 4 v, u, v < R, over k = 0 .. K - 1 (indices clamped into range for the loads; fo stores what lies
// inside).  keep(i0, j0, rows, cols) skips whole tiles.
template <int R, class TM, class FA, class FB, class FM, class FI, class FO, class FK>
__device__ __forceinline__ void warp_tiles_r(const TM &tm, int M, int N, int K, FA fa, FB fb, FM mac, FI init, FO fo,
                                             FK keep) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    const int li = lane & 7, lj = lane >> 3;
    constexpr int TI = 8 * R, TJ = 4 * R;
    const int nti = (M + TI - 1) / TI, ntj = (N + TJ - 1) / TJ;
    for (int idx = warp; idx < nti * ntj; idx += nw) {
        const int i0 = (idx % nti) * TI, j0 = (idx / nti) * TJ;
        if (!keep(i0, j0, TI, TJ)) continue;
        int ii[R], jj[R];
        df_acc acc[R][R];
#pragma unroll
        for (int u = 0; u < R; u++) {
            ii[u] = i0 + li + 8 * u < M ? i0 + li + 8 * u : M - 1;
            jj[u] = j0 + lj + 4 * u < N ? j0 + lj + 4 * u : N - 1;
        }
#pragma unroll
        for (int u = 0; u < R; u++)
#pragma unroll
            for (int v = 0; v < R; v++) acc[u][v] = init(ii[u], jj[v]);
#pragma unroll(R == 2 ? 2 : 1)
        for (int k = 0; k < K; k++) {
            decltype(fa(0, 0)) a[R];
            decltype(fb(0, 0)) b[R];
#pragma unroll
            for (int u = 0; u < R; u++) {
                a[u] = fa(ii[u], k);
                b[u] = fb(k, jj[u]);
            }
#pragma unroll
            for (int u = 0; u < R; u++)
#pragma unroll
                for (int v = 0; v < R; v++) mac(acc[u][v], a[u], b[v]);
        }
#pragma unroll
        for (int u = 0; u < R; u++)
#pragma unroll
            for (int v = 0; v < R; v++)
                if (i0 + li + 8 * u < M && j0 + lj + 4 * v < N) fo(ii[u], jj[v], acc[u][v]);
    }
}

// R = 2, or 4 on a cluster whose warps all get such a tile (half the loads per product: on a cluster the operands come
// through L1, 8 bytes a lane).  An element's arithmetic does not depend on R.
template <class TM, class FA, class FB, class FM, class FI, class FO, class FK>
__device__ __forceinline__ void warp_tiles(const TM &tm, int M, int N, int K, FA fa, FB fb, FM mac, FI init, FO fo,
                                           FK keep) {
    if constexpr (TM::ctas > 1)
        if ((long) ((M + 31) / 32) * ((N + 15) / 16) >= TM::nw()) {
            warp_tiles_r<4>(tm, M, N, K, fa, fb, mac, init, fo, keep);
            return;
        }
    warp_tiles_r<2>(tm, M, N, K, fa, fb, mac, init, fo, keep);
}

// acc += a b for floats, exactly (Ogita, Rump and Oishi's Dot2).
__device__ __forceinline__ void acc_exact(df_acc &acc, float a, float b) {
    const float p = __fmul_rn(a, b), e = __fmaf_rn(a, b, -p);
    const float t = __fadd_rn(acc.s, p), z = __fsub_rn(t, acc.s);
    const float es = __fadd_rn(__fsub_rn(acc.s, __fsub_rn(t, z)), __fsub_rn(p, z));
    acc.s = t;
    acc.e = __fadd_rn(acc.e, __fadd_rn(e, es));
}

// E (rk x rk float-float, ld rk) = J^T J - I of the float J (ld ldj).
template <class TM>
__device__ void ns_gram(const TM &tm, const float *J, int ldj, int rk, df *E) {
    warp_tiles(
        tm, rk, rk, rk, [&](int i, int k) { return J[k + (size_t) i * ldj]; },
        [&](int k, int j) { return J[k + (size_t) j * ldj]; },
        [](df_acc &c, float a, float b) { acc_exact(c, a, b); },
        [](int i, int j) { return df_acc{i == j ? -1.f : 0.f, 0.f}; },
        [&](int i, int j, df_acc c) { E[i + (size_t) j * rk] = df_acc_value(c); }, [](int, int, int, int) { return true; });
}

// Largest column sum of |E| (bounds its norm).
template <class TM>
__device__ float ns_norm(const TM &tm, const df *E, int rk, int *s_bits) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    if (tm.tid == 0) *s_bits = 0;
    tm.sync();
    float top = 0.f;
    for (int j = warp; j < rk; j += nw) {
        float t = 0.f;
        for (int i = lane; i < rk; i += 32) t += fabsf(E[i + (size_t) j * rk].h);
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (!(t <= top)) top = t;
    }
    if (lane == 0) atomicMax(s_bits, __float_as_int(fabsf(top)));  // ordered like its bits, a NaN above all
    tm.sync();
    return __int_as_float(*s_bits);
}

// J64 = J (I + H), written over E (both ld rk), a warp per column.  V (ld ldv): rk x rk floats for
// 3/8 E^2 - 5/16 E^3.  scr: two vectors of rk floats of shared memory (scr_ld apart) for each of the
// first scr_warps warps of a CTA; the other warps wait.
template <class TM>
__device__ void ns_apply(const TM &tm, const float *J, int ldj, int rk, df *E, float *V, int ldv, float *scr,
                         int scr_ld, int scr_warps) {
    const int lane = threadIdx.x & 31;
    const int wpc = tm.warps_per_cta(), wic = tm.warp() % wpc, cta = tm.warp() / wpc, ctas = tm.nw() / wpc;
    const int first = wic < scr_warps ? cta * scr_warps + wic : rk, step = ctas * scr_warps;
    float *s1 = scr + (size_t) (2 * wic) * scr_ld, *s2 = s1 + scr_ld;
    // out_i = sum_l E_il v(l), four rows a lane at a time
    auto apply_e = [&](auto v, auto store) {
        for (int i0 = 0; i0 < rk; i0 += 128) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int l = 0; l < rk; l++) {
                const float vl = v(l);
                const df *El = E + (size_t) l * rk + i0 + lane;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (i0 + lane + 32 * q < rk) acc[q] = fmaf(El[32 * q].h, vl, acc[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (i0 + lane + 32 * q < rk) store(i0 + lane + 32 * q, acc[q]);
        }
    };
    for (int j = first; j < rk; j += step) {
        const df *Ej = E + (size_t) j * rk;
        for (int i = lane; i < rk; i += 32) s2[i] = Ej[i].h;
        __syncwarp();
        apply_e([&](int l) { return s2[l]; }, [&](int i, float y) { s1[i] = 0.375f * s2[i] - 0.3125f * y; });
        __syncwarp();
        apply_e([&](int l) { return s1[l]; }, [&](int i, float y) { V[i + (size_t) j * ldv] = y; });
        __syncwarp();
    }
    tm.sync();
    for (int j = first; j < rk; j += step) {
        df *Ej = E + (size_t) j * rk;
        for (int i = lane; i < rk; i += 32) {
            df m = Ej[i];
            m.h *= -0.5f;
            m.l *= -0.5f;
            const df h = df_add(m, df_f(V[i + (size_t) j * ldv]));
            s1[i] = h.h;
            s2[i] = h.l;
        }
        __syncwarp();
        double *out = reinterpret_cast<double *>(Ej);
        for (int i0 = 0; i0 < rk; i0 += 64) {
            df_acc acc[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 2
            for (int l = 0; l < rk; l++) {
                const float hh = s1[l], hl = s2[l];
                const float *Jl = J + (size_t) l * ldj + i0 + lane;
#pragma unroll
                for (int q = 0; q < 2; q++)
                    if (i0 + lane + 32 * q < rk) {
                        const float a = Jl[32 * q];
                        acc_exact(acc[q], a, hh);
                        acc[q].e = __fmaf_rn(a, hl, acc[q].e);
                    }
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int i = i0 + lane + 32 * q;
                if (i < rk) {
                    const df d = df_acc_value(acc[q]);
                    out[i] = double_scaled_up(J[i + (size_t) j * ldj], 0) +
                             (double_scaled_up(d.h, 0) + double_scaled_up(d.l, 0));
                }
            }
        }
        __syncwarp();
    }
}

// Largest ||J32^T J32 - I||_1 for which the truncated series is exact to working precision.
constexpr float PRECOND_MAX_ORTH = 4e-4f;
constexpr int CORRECT_MAX_PASSES = 4;
constexpr float CORRECT_MAX_TAN = 0.02f;

// Corrections W <- W exp(S) until every pair of columns is orthogonal to tol, W rows x nc (ld rows).
// Wh: float-float copy of W 2^-e_j (ld ldh), T: 2 nc^2 floats (S 2^(e_i - e_j), then S^2 / 2 likewise),
// nrm / ex: a float-float norm and an exponent per column.  Columns below the noise floor of the FP64 sweeps
// are left alone, as there.  Returns whether the columns are orthogonal to tol.
template <class TM>
__device__ bool jacobi_correct(const TM &tm, double *W, int rows, int nc, df *Wh, int ldh, float *T, df *nrm, int *ex,
                               int *s_cos, int *s_tan, float tol, int *passes) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    float *S = T, *Q = T + (size_t) nc * nc;
    for (int pass = 0; pass < CORRECT_MAX_PASSES; pass++) {
        // columns as float-float values near 1 and their squared norms
        for (int j = warp; j < nc; j += nw) {
            const double *w = W + (size_t) j * rows;
            int e = 0;
            for (int r = lane; r < rows; r += 32) {
                const int f = (int) ((__double_as_longlong(w[r]) >> 52) & 0x7ff);
                e = e > f ? e : f;
            }
            for (int o = 16; o > 0; o >>= 1) {
                const int f = __shfl_xor_sync(0xffffffffu, e, o);
                e = e > f ? e : f;
            }
            e = e ? e - 1023 : -1022;
            df sq = df_f(0.f);
            for (int r = lane; r < rows; r += 32) {
                const df v = df_scaled_down(w[r], e);
                Wh[r + (size_t) j * ldh] = v;
                sq = df_fma(v, v, sq);
            }
            sq = df_group_sum(sq, 32);
            if (lane == 0) {
                nrm[j] = sq;
                ex[j] = e;
            }
        }
        if (tm.tid == 0) {
            *s_cos = 0;
            *s_tan = 0;
        }
        tm.sync();
        // the noise floor relative to the largest column (uniform: every thread scans the same norms)
        int etop = -2000;
        for (int j = lane; j < nc; j += 32)
            if (nrm[j].h > 0.f && ex[j] > etop) etop = ex[j];
        for (int o = 16; o > 0; o >>= 1) {
            const int f = __shfl_xor_sync(0xffffffffu, etop, o);
            etop = etop > f ? etop : f;
        }
        float top = 0.f;
        for (int j = lane; j < nc; j += 32)
            if (ex[j] - etop >= -60) {
                const float v = ldexpf(nrm[j].h, 2 * (ex[j] - etop));
                top = top > v ? top : v;
            }
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float noise = 2.220446e-16f * (float) rows;
        auto live = [&](int j) {
            const int d = ex[j] - etop;
            return d >= -60 && ldexpf(nrm[j].h, 2 * d) > top * noise * noise;
        };
        float mcos = 0.f, mtan = 0.f;
        warp_tiles(
            tm, nc, nc, rows, [&](int i, int k) { return Wh[k + (size_t) i * ldh]; },
            [&](int k, int j) { return Wh[k + (size_t) j * ldh]; },
            [](df_acc &c, df a, df b) { df_acc_fma(c, a, b); }, [](int, int) { return df_acc{0.f, 0.f}; },
            [&](int i, int j, df_acc cc) {
                if (i > j) return;
                if (i == j) {
                    S[i + (size_t) i * nc] = 0.f;
                    return;
                }
                const df c = df_acc_value(cc);
                const df a = nrm[i], b = nrm[j];
                const int d = ex[j] - ex[i];
                float tt = 0.f;
                const float cosine = fabsf(c.h) * rsqrtf(a.h) * rsqrtf(b.h);
                if (d >= -60 && d <= 60 && live(i) && live(j) && cosine > 0.1f * tol) {
                    // in units of the larger column: b' = b 4^d, c' = c 2^d (or a' = a 4^-d, c' = c 2^-d)
                    const int da = d > 0 ? -d : 0, db = d > 0 ? 0 : d;
                    df as, bs;
                    as.h = ldexpf(a.h, 2 * da);
                    as.l = ldexpf(a.l, 2 * da);
                    bs.h = ldexpf(b.h, 2 * db);
                    bs.l = ldexpf(b.l, 2 * db);
                    const float zeta = df_add(bs, -as).h / (2.f * ldexpf(c.h, d > 0 ? -d : d));
                    tt = rotation_tangent(zeta);
                    mcos = fmaxf(mcos, cosine);
                    mtan = fmaxf(mtan, fabsf(tt));
                }
                S[i + (size_t) j * nc] = ldexpf(tt, -d);
                S[j + (size_t) i * nc] = -ldexpf(tt, d);
            },
            [](int i0, int j0, int, int tj) { return i0 <= j0 + tj - 1; });
        for (int o = 16; o > 0; o >>= 1) {
            mcos = fmaxf(mcos, __shfl_xor_sync(0xffffffffu, mcos, o));
            mtan = fmaxf(mtan, __shfl_xor_sync(0xffffffffu, mtan, o));
        }
        if (lane == 0) {
            atomicMax(s_cos, __float_as_int(mcos));
            atomicMax(s_tan, __float_as_int(mtan));
        }
        tm.sync();
        mcos = __int_as_float(*s_cos);
        mtan = __int_as_float(*s_tan);
        *passes = pass + 1;
        if (mcos <= tol) return true;
        if (!(mtan < CORRECT_MAX_TAN)) return false;
        const bool second = (float) nc * mtan * mtan > 1e-17f;  // else S^2 / 2 is below rounding
        if (second) {
            warp_tiles(
                tm, nc, nc, nc, [&](int i, int k) { return S[i + (size_t) k * nc]; },
                [&](int k, int j) { return S[k + (size_t) j * nc]; },
                [](df_acc &c, float a, float b) { c.s = fmaf(a, b, c.s); }, [](int, int) { return df_acc{0.f, 0.f}; },
                [&](int i, int j, df_acc c) { Q[i + (size_t) j * nc] = 0.5f * c.s; }, [](int, int, int, int) { return true; });
            tm.sync();
        }
        warp_tiles(
            tm, rows, nc, nc, [&](int i, int k) { return Wh[i + (size_t) k * ldh]; },
            [&](int k, int j) {
                df t;
                t.h = S[k + (size_t) j * nc];
                t.l = second ? Q[k + (size_t) j * nc] : 0.f;
                return t;
            },
            [](df_acc &c, df a, df b) { df_acc_fma(c, a, b); }, [](int, int) { return df_acc{0.f, 0.f}; },
            [&](int i, int j, df_acc c) {
                const df d = df_acc_value(c);
                double *w = W + i + (size_t) j * rows;
                *w += double_scaled_up(d.h, ex[j]) + double_scaled_up(d.l, ex[j]);  // the inner sum is exact
            },
            [](int, int, int, int) { return true; });
        tm.sync();
        // what is left after the correction: second order in the angles
        if ((float) nc * mtan * mcos < 0.1f * tol) return true;
    }
    return false;
}


// The cross steps of a block pair with the first block's columns in registers (RQ quads a lane, CPG columns a group of
// G lanes): only the second block's columns go through shared memory, once per step.  The steps are bound by
// shared-memory bandwidth: 3,400 cycles each for 22 + 22 columns of 340 rows when both go through it twice.
// Same operations as jacobi32_block_pair.
template <int G, int RQ, int CPG, class TM>
__device__ int jacobi32_cross(const TM &tm, float4 *Y, int ls4, int x4, int j4, int nc_a, int nc_b, int off_b, float tol) {
    const int gl = tm.tid % G, grp = tm.tid / G;
    constexpr int NG = TM::nth / G;
    const int wide = nc_a > nc_b ? nc_a : nc_b, len = x4 + j4;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 x[CPG][RQ];
#pragma unroll
    for (int c = 0; c < CPG; c++)
#pragma unroll
        for (int u = 0; u < RQ; u++) {
            const int r = gl + G * u, p = grp + c * NG;
            x[c][u] = p < nc_a && r < len ? Y[(size_t) p * ls4 + r] : zero;
        }
    int rotations = 0;
    for (int t = 0; t < wide; t++) {
#pragma unroll
        for (int c = 0; c < CPG; c++) {
            const int p = grp + c * NG, q = p + t < wide ? p + t : p + t - wide;
            const bool act = p < nc_a && q < nc_b;
            float4 *yc = Y + (size_t) (off_b + (act ? q : 0)) * ls4;
            float4 y[RQ];
            float a = 0.f, b = 0.f, d = 0.f;
#pragma unroll
            for (int u = 0; u < RQ; u++) {
                const int r = gl + G * u;
                y[u] = act && r < len ? yc[r] : zero;
                if (r < x4) {
                    const float4 e = x[c][u], f = y[u];
                    a = fmaf(e.x, e.x, fmaf(e.y, e.y, fmaf(e.z, e.z, fmaf(e.w, e.w, a))));
                    b = fmaf(f.x, f.x, fmaf(f.y, f.y, fmaf(f.z, f.z, fmaf(f.w, f.w, b))));
                    d = fmaf(e.x, f.x, fmaf(e.y, f.y, fmaf(e.z, f.z, fmaf(e.w, f.w, d))));
                }
            }
#pragma unroll
            for (int o = G >> 1; o > 0; o >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
                d += __shfl_xor_sync(0xffffffffu, d, o);
            }
            if (act && a > 0.f && b > 0.f && fabsf(d) * rsqrtf(a) * rsqrtf(b) > tol) {
                float cs, sn;
                rotation32(a, b, d, cs, sn);
#pragma unroll
                for (int u = 0; u < RQ; u++) {
                    const int r = gl + G * u;
                    const float4 e = x[c][u], f = y[u];
                    x[c][u] = make_float4(fmaf(cs, e.x, -sn * f.x), fmaf(cs, e.y, -sn * f.y), fmaf(cs, e.z, -sn * f.z),
                                          fmaf(cs, e.w, -sn * f.w));
                    if (r < len)
                        yc[r] = make_float4(fmaf(cs, f.x, sn * e.x), fmaf(cs, f.y, sn * e.y), fmaf(cs, f.z, sn * e.z),
                                            fmaf(cs, f.w, sn * e.w));
                }
                rotations += gl == 0;
            }
        }
        tm.sync();
    }
#pragma unroll
    for (int c = 0; c < CPG; c++)
#pragma unroll
        for (int u = 0; u < RQ; u++) {
            const int r = gl + G * u, p = grp + c * NG;
            if (p < nc_a && r < len) Y[(size_t) p * ls4 + r] = x[c][u];
        }
    tm.sync();
    return rotations;
}

// Columns of the preconditioner's working matrix (x4 quads of X above j4 of J): a length of 4 mod 8 quads, so that two
// 4-lane groups, a quarter-warp, meet no bank conflict.
__host__ __device__ constexpr int precond_quads(int x4, int j4) { return ((x4 + j4 + 3) & ~7) + 4; }

// Stack width up to which a core gets eight lanes a pair from 33 columns on, and not from 65: about a quarter of an SM's
// shared memory.  A width, not the team that a launch gives the update.
constexpr int SMALL_K = 82;
constexpr int SWEEP_BLOCKS = 2 * WIDE_CTAS;  // column blocks of a core that a cluster can hold two at a time a CTA
constexpr int BLOCK_G16_QUADS = 42;          // up to 168 rows (and as many columns, eleven a block)

// Column blocks of the cluster's sweeps: every CTA of the cluster holds one pair of blocks at a time in its
// shared memory (buf, `quads` float4s) and sweeps the pairs of columns that it gives; the blocks meet in
// round-robin order, through global memory (Y, columns of x4 + j4 quads).
template <class TM>
__device__ int jacobi32_blocks(const TM &tm, float4 *Y, int x4, int j4, int nc, float4 *buf, int quads, float tol) {
    const int L = x4 + j4;
    int nblk = 0, w = 0;
    do {
        nblk += 2 * TM::ctas;
        w = (nc + nblk - 1) / nblk;
    } while (w > 1 && 2 * w * L > quads);
    const Team<TM::cta_threads> ct{(int) threadIdx.x, 1};
    const bool rows_g16 = x4 <= BLOCK_G16_QUADS;  // cores that one SM can hold: the lanes per pair it takes
    int rot = 0;
    for (int t = 0; t < nblk - 1; t++) {
        for (int pp = tm.rank; pp < nblk / 2; pp += TM::ctas) {
            int bi, bj;
            jacobi_pair(t, pp, nblk, bi, bj);
            const int ra = nc - bi * w, rb = nc - bj * w;
            const int na = ra < 0 ? 0 : (ra < w ? ra : w), nb = rb < 0 ? 0 : (rb < w ? rb : w);
            if (na + nb < 2 || (t > 0 && (na == 0 || nb == 0))) continue;
            float4 *ya = Y + (size_t) bi * w * L, *yb = Y + (size_t) bj * w * L;
            for (int e = threadIdx.x; e < na * L; e += TM::cta_threads) buf[e] = __ldcg(ya + e);
            for (int e = threadIdx.x; e < nb * L; e += TM::cta_threads) buf[w * L + e] = __ldcg(yb + e);
            ct.sync();
            if (rows_g16) {
                if (t > 0) rot += jacobi32_cross<16, 6, 1>(ct, buf, L, x4, j4, na, nb, w, tol);
                else rot += jacobi32_block_pair<16>(ct, buf, L, x4, j4, na, nb, w, false, tol);
            } else if (t > 0 && L <= 6 * 32 && w <= 16) {
                rot += jacobi32_cross<32, 6, 1>(ct, buf, L, x4, j4, na, nb, w, tol);
            } else if (t > 0 && L <= 6 * 32 && w <= 32) {
                rot += jacobi32_cross<32, 6, 2>(ct, buf, L, x4, j4, na, nb, w, tol);
            } else if (t > 0 && L <= 8 * 32 && w <= 16) {
                rot += jacobi32_cross<32, 8, 1>(ct, buf, L, x4, j4, na, nb, w, tol);
            } else {
                rot += jacobi32_block_pair<32>(ct, buf, L, x4, j4, na, nb, w, t > 0, tol);
            }
            for (int e = threadIdx.x; e < na * L; e += TM::cta_threads) ya[e] = buf[e];
            for (int e = threadIdx.x; e < nb * L; e += TM::cta_threads) yb[e] = buf[w * L + e];
            ct.sync();
        }
        tm.sync();
    }
    return rot;
}

// Steps 1-3 and the corrections for X (rows x nc, lower trapezoidal, ld ldx).  Scratch: y (quads float4s, for
// a cluster in global memory) and for a cluster buf (shared memory); E64 (nc^2 doubles), W (rows x nc
// doubles; may lie over y in global memory), Wh (rows x nc float-float values, ld ldh; may lie over y in
// shared memory and over X), V (floats, ldv; unused entries of y or memory of its own).  On return W holds
// the columns; *converged as for the sweeps.  Returns false with X untouched when J32 is no rotation.
struct PrecondBuffers {
    float4 *y;
    int ls4;           // quads per column of y
    int blocks;        // column blocks of the sweep order (0: round robin)
    bool g8;           // round robin: eight lanes a pair, not four
    float4 *buf;       // cluster: shared memory for a pair of blocks and the vectors of ns_apply
    int buf_quads;
    double *e64;
    double *w;
    df *wh;
    int ldh;
    float *v;
    int ldv;
};

template <class TM>
__device__ bool jacobi_precond(const TM &tm, const double *X, int ldx, int rows, int nc, const PrecondBuffers &b,
                               df *nrm, int *ex, int *s_rot, int *s_emax, int *s_cos, int *s_tan, float tol,
                               int *sweeps, bool *converged) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    const int lr = lane >> 2, lc = lane & 3;
    const int x4 = (rows + 3) >> 2, j4 = (nc + 3) >> 2;
    float *Y = reinterpret_cast<float *>(b.y);
    const int ldy = 4 * b.ls4;
    if (tm.tid == 0) *s_emax = 0;
    tm.sync();
    int em = 0;
    for (int j = warp; j < nc; j += nw)
        for (int r = lane; r < rows; r += 32) {
            const int f = (int) ((__double_as_longlong(X[r + (size_t) j * ldx]) >> 52) & 0x7ff);
            em = em > f ? em : f;
        }
    atomicMax(s_emax, em);
    tm.sync();
    const int esc = *s_emax ? *s_emax - 1023 : 0;
    for (int j = warp; j < nc; j += nw) {
        float *y = Y + (size_t) j * ldy;
        for (int r = lane; r < 4 * x4; r += 32) y[r] = r < rows ? df_scaled_down(X[r + (size_t) j * ldx], esc).h : 0.f;
        for (int r = lane; r < 4 * j4; r += 32) y[4 * x4 + r] = r == j ? 1.f : 0.f;
    }
    tm.sync();
    // 1. single-precision sweeps, until one turns few pairs: what it leaves is second order
    for (int s = 0; s < PRECOND_MAX_SWEEPS; s++) {
        if (tm.tid == 0) *s_rot = 0;
        tm.sync();
        int rot;
        if constexpr (TM::ctas > 1) rot = jacobi32_blocks(tm, b.y, x4, j4, nc, b.buf, b.buf_quads, PRECOND_TOL32);
        else if (b.blocks) rot = jacobi32_sweep<16>(tm, b.y, b.ls4, x4, j4, nc, b.blocks, PRECOND_TOL32);
        else if (b.g8) rot = jacobi32_sweep<8>(tm, b.y, b.ls4, x4, j4, nc, 0, PRECOND_TOL32);
        else rot = jacobi32_sweep<4>(tm, b.y, b.ls4, x4, j4, nc, 0, PRECOND_TOL32);
        if (rot) atomicAdd(s_rot, rot);
        tm.sync();
        const int total = *s_rot;
        tm.sync();
        ++*sweeps;
        if (total * 16 <= nc * (nc - 1) / 2) break;
    }
    // 2. the orthogonal factor of J32
    const float *J = Y + 4 * x4;
    df *E = reinterpret_cast<df *>(b.e64);
    ns_gram(tm, J, ldy, nc, E);
    tm.sync();
    if (!(ns_norm(tm, E, nc, s_rot) < PRECOND_MAX_ORTH)) return false;
    if constexpr (TM::ctas > 1) {
        float *scr = reinterpret_cast<float *>(b.buf);
        const int fit = 4 * b.buf_quads / (2 * nc), wpc = tm.warps_per_cta();
        ns_apply(tm, J, ldy, nc, E, b.v, b.ldv, scr, nc, fit < wpc ? fit : wpc);
    } else {
        ns_apply(tm, J, ldy, nc, E, b.v, b.ldv, Y, ldy, nc / 2 < nw ? nc / 2 : nw);  // over X32, which is done
    }
    tm.sync();
    // 3. W = X J on DMMA; column l of X starts at row l
    const double *J64 = b.e64;
    const int ntr = (rows + 7) >> 3, ntc = (nc + 7) >> 3;
    for (int idx = warp; idx < ntr * ntc; idx += nw) {
        const int tr = idx % ntr, tc = idx / ntr;
        const int irow = tr * 8 + lr, icol = tc * 8 + lr;
        const int kend = nc < tr * 8 + 8 ? nc : tr * 8 + 8;
        const double *jc = J64 + (size_t) (icol < nc ? icol : 0) * nc;
        double d0 = 0.0, d1 = 0.0;
#pragma unroll 4
        for (int l4 = 0; l4 < kend; l4 += 4) {
            const int l = l4 + lc;
            const double av = (irow < rows && l < nc) ? X[irow + (size_t) l * ldx] : 0.0;
            const double bv = (icol < nc && l < nc) ? jc[l] : 0.0;
            dmma(d0, d1, av, bv);
        }
        const int col = tc * 8 + 2 * lc;
        if (irow < rows && col < nc) b.w[irow + (size_t) col * rows] = d0;
        if (irow < rows && col + 1 < nc) b.w[irow + (size_t) (col + 1) * rows] = d1;
    }
    tm.sync();
    int passes = 0;
    *converged = jacobi_correct(tm, b.w, rows, nc, b.wh, b.ldh, reinterpret_cast<float *>(b.e64), nrm, ex, s_cos, s_tan,
                                tol, &passes);
    *sweeps += passes;
    return true;
}

// A step's reflector H = I - tau v v^T for the pivot column x (rows s ..), v = [1; scale x_{s+1}, ..] (dlarfg's
// beta and tau; x stays as it is: only R is kept).  sigma = ||x_{s+1..}||^2.  One reciprocal square root and one
// reciprocal: every FP64 instruction of this chain holds up the whole team.  tau and scale stay in range
// wherever sigma is not zero; 2 / ||x||^2 in one number, an instruction less a column, overflows for columns
// below 7e-155.
struct Reflector {
    double beta, tau, scale;
};
__device__ __forceinline__ Reflector make_reflector(double alpha, double sigma) {
    Reflector h{alpha, 0.0, 0.0};
    if (sigma != 0.0) {
        const double q = fma(alpha, alpha, sigma), r = rsqrt(q), nrm = q * r;
        h.beta = -copysign(nrm, alpha);
        h.tau = fma(fabs(alpha), r, 1.0);                            // (beta - alpha) / beta
        h.scale = copysign(__drcp_rn(nrm + fabs(alpha)), alpha);     // 1 / (alpha - beta)
    }
    return h;
}

// One step of the pivoted QR: H applied to column y (rows s .. mrows - 1) by a group of G lanes, its squared norm
// below row s downdated and recomputed exactly when the downdate loses four or more digits (LAPACK
// dlaqp2's guard).  act: whether the group has a column (uniform in the group); every lane of the warp calls.
template <int G>
__device__ __forceinline__ void reflect_column(bool act, double *y, const double *x, const Reflector &h, int s,
                                               int mrows, int gl, double *nrm, double *nref) {
    double w = 0.0;
    if (act && h.tau != 0.0)
        for (int i = s + 1 + gl; i < mrows; i += G) w = fma(x[i], y[i], w);
    w = group_sum(w, G);
    double ys = 0.0;
    if (act) {
        ys = y[s];  // every lane of the group reads the old y[s] before lane 0 writes it
        if (h.tau != 0.0) {
            w = fma(w, h.scale, ys) * h.tau;
            ys -= w;
            const double t = w * h.scale;
            for (int i = s + 1 + gl; i < mrows; i += G) y[i] = fma(-t, x[i], y[i]);
        }
    }
    __syncwarp();
    double nn = 0.0;
    bool exact = false;
    if (act) {
        if (gl == 0) y[s] = ys;
        nn = fma(-ys, ys, *nrm);
        exact = !(nn > 1e-8 * *nref);
    }
    if (__any_sync(0xffffffffu, exact)) {
        double e = 0.0;
        if (exact)
            for (int i = s + 1 + gl; i < mrows; i += G) e = fma(y[i], y[i], e);
        e = group_sum(e, G);
        if (exact) nn = e;
    }
    __syncwarp();
    if (act && gl == 0) {
        *nrm = nn;
        if (exact) *nref = nn;
    }
}

// (value, index) with the largest value over a warp, ties to the lower index; values are the bits of
// non-negative doubles, ordered like them, a NaN above all.  A norm that is not finite is the first pivot, whose
// reflector makes every column NaN; behind the first step it ends the factorisation (a core with a NaN or
// an infinity gives a rank-1 tile of NaN).
constexpr long long NRM_INF_BITS = 0x7ff0000000000000LL, NRM_SIGN_MASK = 0x7fffffffffffffffLL;
__device__ __forceinline__ void warp_argmax(long long &v, int &i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) {
            v = ov;
            i = oi;
        }
    }
}

// Householder QR with column pivoting of A (mrows x ncols, ld lda), stopped early once
// every remaining column is below sqrt(stop2) in norm (LAPACK dgeqp3 semantics for the part that
// is computed: A P = Q R).  stop2 < 0 disables the early stop; stop2 == 0 with rel > 0 sets
// stop2 = (rel * |r_00|)^2 after the first pivot.  Columns stay in place: pvt[s] is the column of step s,
// R(s, t) stands in A(s, pvt[t]).  Returns the number of rows of R that were computed.
// Two barriers a step: the first warp picks the pivot and forms the reflector, the team applies it.
template <int G, class TM>
__device__ int qrcp_steps(const TM &tm, double *A, int lda, int mrows, int ncols, double stop2, double rel, double *nrm,
                          double *nref, int *pvt, double *red, int *redi) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int CPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    for (int j = warp; j < ncols; j += nw) {
        const double *col = A + (size_t) j * lda;
        double t = 0.0;
        for (int i = lane; i < mrows; i += 32) t = fma(col[i], col[i], t);
        t = warp_sum(t);
        if (lane == 0) nrm[j] = nref[j] = t;
    }
    for (int j = tm.tid; j < ncols; j += tm.nth) pvt[j] = j;
    tm.sync();
    const int kk = mrows < ncols ? mrows : ncols;
    double lim = stop2;
    int rk = kk;
    for (int s = 0; s < kk; s++) {
        if (warp == 0) {
            long long bv = -1;
            int bi = ncols, at = s;  // the largest norm's column (ties to the lower one) and its place in pvt
            for (int j = s + lane; j < ncols; j += 32) {
                const int c = pvt[j];
                const long long v = __double_as_longlong(nrm[c]) & NRM_SIGN_MASK;
                if (v > bv || (v == bv && c < bi)) {
                    bv = v;
                    bi = c;
                    at = j;
                }
            }
            {
                const int mine = bi;
                warp_argmax(bv, bi);
                at = __shfl_sync(0xffffffffu, at, __ffs(__ballot_sync(0xffffffffu, mine == bi)) - 1);
            }
            const double top = bv < 0 ? 0.0 : __longlong_as_double(bv);
            if (s == 0 && stop2 == 0.0 && rel > 0.0) lim = rel * rel * top;
            const bool stop = bv >= NRM_INF_BITS ? s > 0 : (top <= lim || top <= 0.0);
            if (!stop) {
                const int cs = bi;
                __syncwarp();
                if (lane == 0) {
                    pvt[at] = pvt[s];
                    pvt[s] = cs;
                }
                double *x = A + (size_t) cs * lda;
                double t = 0.0;
                for (int i = s + 1 + lane; i < mrows; i += 32) t = fma(x[i], x[i], t);
                t = warp_sum(t);
                const Reflector h = make_reflector(x[s], t);
                __syncwarp();
                if (lane == 0) {
                    red[0] = h.tau;
                    red[1] = h.scale;
                    x[s] = h.beta;
                    redi[1] = cs;
                }
            }
            if (lane == 0) redi[0] = stop;
        }
        tm.sync();
        if (redi[0]) {
            rk = s;
            break;
        }
        const Reflector h{0.0, red[0], red[1]};
        const double *x = A + (size_t) redi[1] * lda;
        for (int j0 = s + 1 + warp * CPW; j0 < ncols; j0 += nw * CPW) {
            const int j = j0 + grp;
            const bool act = j < ncols;
            const int c = pvt[act ? j : s];
            reflect_column<G>(act, A + (size_t) c * lda, x, h, s, mrows, gl, nrm + c, nref + c);
        }
        tm.sync();
    }
    // the columns never chosen, in ascending order (at most one a thread: a team has more threads than columns)
    const int j = rk + tm.tid;
    int c = 0, pos = rk;
    if (j < ncols) {
        c = pvt[j];
        for (int t = rk; t < ncols; t++) pos += pvt[t] < c;
    }
    tm.sync();
    if (j < ncols) pvt[pos] = c;
    tm.sync();
    return rk;
}

// Columns of up to 64, 256 or more rows are handled by groups of 4, 8 or 16 lanes, several columns per warp
// instruction, so the reductions and the per-column scalar work are shared.
template <class TM>
__device__ int qrcp_truncated(const TM &tm, double *A, int lda, int mrows, int ncols, double stop2, double rel, double *nrm,
                              double *nref, int *pvt, double *red, int *redi) {
    if (mrows <= 64) return qrcp_steps<4>(tm, A, lda, mrows, ncols, stop2, rel, nrm, nref, pvt, red, redi);
    if (mrows <= 256) return qrcp_steps<8>(tm, A, lda, mrows, ncols, stop2, rel, nrm, nref, pvt, red, redi);
    return qrcp_steps<16>(tm, A, lda, mrows, ncols, stop2, rel, nrm, nref, pvt, red, redi);
}

// The same for a cluster: column j lives in the shared memory of CTA j % CTAS, and a step costs one
// cluster barrier: every CTA offers its best column to all, each reads the winner's column from its owner and
// forms the reflector itself.  (Through global memory a step took 24,000 cycles on a 130-column core, bound
// by dependent L2 round trips and five cluster barriers.)  R goes to X = R^T directly (rk columns of
// ncols entries, ld ldx, entry t of column s for pivot order t).  pvt: shared by the cluster.
// Doubles beside the columns.
__device__ __forceinline__ int qrcp_cluster_aux(int mrows, int ncols, int ctas) {
    const int nl = (ncols + ctas - 1) / ctas;
    return 3 * nl + 2 * mrows + (ncols + 1) / 2 + 6 * ctas + 8;
}

template <int G, class TM>
__device__ int qrcp_cluster(const TM &tm, const double *M, int ldm, int mrows, int ncols, double stop2, double rel,
                            double *X, int ldx, int *pvt, double *pool, int pool_doubles, double *spill, int lds) {
    constexpr int C = TM::ctas, CPW = 32 / G;
    const Team<TM::cta_threads> ct{(int) threadIdx.x, 1};
    const int warp = ct.warp(), lane = threadIdx.x & 31, nw = ct.nw(), rank = tm.rank;
    const int gl = lane % G, grp = lane / G;
    const int nlmax = (ncols + C - 1) / C, nl = rank < ncols ? (ncols - rank + C - 1) / C : 0;
    // local column q is column rank + q C; the first `fit` in shared memory, the others in place in `spill`
    double *A = pool;
    const int room = (pool_doubles - qrcp_cluster_aux(mrows, ncols, C)) / mrows, fit = room < nlmax ? room : nlmax;
    auto column = [&](int r, int q) { return spill + (size_t) (r + q * C) * lds; };
    double *nrm = A + (size_t) mrows * fit;
    double *nref = nrm + nlmax;
    double *xb = nref + nlmax;                      // the pivot column
    double *diag = xb + mrows;                      // beta of every step
    double *red = diag + mrows;                     // tau, scale
    long long *cv = reinterpret_cast<long long *>(red + 4);  // candidates of the CTAs, two steps' worth
    int *ci = reinterpret_cast<int *>(cv + 2 * C);
    int *act_list = ci + 2 * C;                     // local columns not chosen yet
    int *taken = act_list + 2 * nlmax;              // per column: chosen (for the leftovers)
    for (int q = warp; q < nl; q += nw) {
        const double *col = M + (size_t) (rank + q * C) * ldm;
        double *own = q < fit ? A + (size_t) q * mrows : column(rank, q);
        double t = 0.0;
        for (int i = lane; i < mrows; i += 32) {
            const double v = col[i];
            own[i] = v;
            t = fma(v, v, t);
        }
        t = warp_sum(t);
        if (lane == 0) nrm[q] = nref[q] = t;
    }
    for (int q = threadIdx.x; q < nl; q += TM::cta_threads) act_list[q] = q;
    for (int j = threadIdx.x; j < ncols; j += TM::cta_threads) taken[j] = 0;
    ct.sync();
    int nact = nl, rk = mrows < ncols ? mrows : ncols;
    const int kk = rk;
    double lim = stop2;
    for (int s = 0; s < kk; s++) {
        const int par = (s & 1) * C;
        if (warp == 0) {
            long long bv = -1;
            int bi = ncols;
            for (int q = lane; q < nact; q += 32) {
                const int c = act_list[q], j = rank + c * C;
                const long long v = __double_as_longlong(nrm[c]) & NRM_SIGN_MASK;
                if (v > bv || (v == bv && j < bi)) {
                    bv = v;
                    bi = j;
                }
            }
            warp_argmax(bv, bi);
            if (lane < C) {
                cluster_map(cv, lane)[par + rank] = bv;
                cluster_map(ci, lane)[par + rank] = bi;
            }
        }
        tm.sync();
        long long bv = lane < C ? cv[par + lane] : -1;
        int bi = lane < C ? ci[par + lane] : ncols;
        warp_argmax(bv, bi);
        const double top = bv < 0 ? 0.0 : __longlong_as_double(bv);
        if (s == 0 && stop2 == 0.0 && rel > 0.0) lim = rel * rel * top;
        if (bv >= NRM_INF_BITS ? s > 0 : (top <= lim || top <= 0.0)) {
            rk = s;
            break;
        }
        const int owner = bi % C, lcol = bi / C;
        if (warp == 0) {
            const double *x = lcol < fit ? cluster_map(A, owner) + (size_t) lcol * mrows : column(owner, lcol);
            double t = 0.0;
            if (lane == 0) xb[s] = x[s];
            for (int i = s + 1 + lane; i < mrows; i += 32) {
                const double v = x[i];
                xb[i] = v;
                t = fma(v, v, t);
            }
            t = warp_sum(t);
            __syncwarp();
            const Reflector h = make_reflector(xb[s], t);
            if (lane == 0) {
                red[0] = h.tau;
                red[1] = h.scale;
                diag[s] = h.beta;
                taken[bi] = 1;
                if (rank == 0) pvt[s] = bi;
            }
        }
        if (owner == rank) {  // drop it from the list (any order will do)
            if (warp == 1) {
                for (int q = lane; q < nact - 1; q += 32)
                    if (act_list[q] == lcol) act_list[q] = act_list[nact - 1];
            }
            nact--;
        }
        ct.sync();
        const Reflector h{0.0, red[0], red[1]};
        for (int q0 = warp * CPW; q0 < nact; q0 += nw * CPW) {
            const bool act = q0 + grp < nact;
            const int c = act_list[act ? q0 + grp : 0];
            reflect_column<G>(act, c < fit ? A + (size_t) c * mrows : column(rank, c), xb, h, s, mrows, gl, nrm + c, nref + c);
        }
        ct.sync();
    }
    ct.sync();
    if (rank == 0 && threadIdx.x == 0) {
        int t = rk;
        for (int j = 0; j < ncols; j++)
            if (!taken[j]) pvt[t++] = j;
    }
    tm.sync();
    for (int t = tm.warp(); t < ncols; t += tm.nw()) {
        const int j = pvt[t];
        const double *col = j / C < fit ? cluster_map(A, j % C) + (size_t) (j / C) * mrows : column(j % C, j / C);
        for (int i = lane; i < rk; i += 32) X[t + (size_t) i * ldx] = i < t ? col[i] : (i == t ? diag[i] : 0.0);
        if (rk == 0 && lane == 0) X[t] = M[(size_t) j * ldm];
    }
    tm.sync();
    return rk;
}

// qrcp_apply in float-float arithmetic (mixed form): H applied to columns s+1 .. ncols-1 by groups of
// G lanes with Dot2 accumulation, squared norms downdated and recomputed when the downdate cancels.
template <int G, class TM>
__device__ __forceinline__ void qrcp_apply_df(const TM &tm, df *A, int lda, int mrows, int ncols, int s, const df *x,
                                              df tau, df *nrm, df *nref) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    constexpr int CPW = 32 / G;
    const int gl = lane % G, grp = lane / G;
    const bool has_tau = tau.h != 0.f;
    for (int j0 = s + 1 + warp * CPW; j0 < ncols; j0 += nw * CPW) {
        const int j = j0 + grp;
        const bool act = j < ncols;
        df *y = A + (size_t) (act ? j : s) * lda;  // idle groups read column s and write nothing
        df w = df_f(0.f);
        if (has_tau) {
            df_acc wa = df_acc_init(gl == 0 ? y[s] : df_f(0.f));
            for (int i = s + 1 + gl; i < mrows; i += G) df_acc_fma(wa, x[i], y[i]);
            w = df_mul(group_sum(df_acc_value(wa), G), tau);
            const df mw = -w;
            if (act)
                for (int i = s + 1 + gl; i < mrows; i += G) y[i] = df_fma(mw, x[i], y[i]);
        }
        const df ys = df_add(y[s], -w);  // every lane of the group reads the old y[s] before lane 0 writes it
        __syncwarp();
        if (act && gl == 0) y[s] = ys;
        df nn = act ? df_add(nrm[j], -df_mul(ys, ys)) : df_f(0.f);
        const bool exact = act && !(nn.h > 1e-8f * nref[j].h);  // lost 4+ digits since the last exact value
        if (__any_sync(0xffffffffu, exact)) {
            df e = df_f(0.f);
            if (exact)
                for (int i = s + 1 + gl; i < mrows; i += G) e = df_fma(y[i], y[i], e);
            e = group_sum(e, G);
            if (exact) nn = e;
        }
        __syncwarp();
        if (act && gl == 0) {
            nrm[j] = nn;
            if (exact) nref[j] = nn;
        }
    }
}

// Float-float version of qrcp_truncated (mixed form), on a matrix scaled so that its entries are
// near 1: same pivoting, early stop (stop2 on squared norms; stop2 == 0 with rel2 > 0 sets
// stop2 = rel2 * |r_00|^2 after the first pivot; stop2 < 0 disables it) and norm downdating with
// exact recomputation when a downdate cancels.  Pivot keys are the float norms' bit patterns
// (non-negative floats order like their bits; a NaN above all, as in the FP64 form).
template <class TM>
__device__ int qrcp_truncated_df(const TM &tm, df *A, int lda, int mrows, int ncols, float stop2, float rel2, df *nrm, df *nref,
                                 int *pvt, float *red, int *redi) {
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    for (int j = warp; j < ncols; j += nw) {
        const df *col = A + (size_t) j * lda;
        df t = df_f(0.f);
        for (int i = lane; i < mrows; i += 32) t = df_fma(col[i], col[i], t);
        t = group_sum(t, 32);
        if (lane == 0) nrm[j] = nref[j] = t;
    }
    for (int j = tm.tid; j < ncols; j += tm.nth) pvt[j] = j;
    tm.sync();
    const int kk = mrows < ncols ? mrows : ncols;
    int rkeep = kk;
    for (int s = 0; s < kk; s++) {
        int bv = -1, bi = s;  // float bits of the largest remaining squared norm (first warp only)
        if (warp == 0) {
            for (int j = s + lane; j < ncols; j += 32) {
                const int v = __float_as_int(nrm[j].h) & 0x7fffffff;
                if (v > bv) {
                    bv = v;
                    bi = j;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const int ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if (lane == 0) {
                redi[64] = bv;
                redi[65] = bi;
                if (s == 0) red[33] = (stop2 == 0.f && rel2 > 0.f) ? rel2 * __int_as_float(bv) : stop2;
            }
        }
        tm.sync();
        const float bvf = __int_as_float(redi[64]);
        bi = redi[65];
        const float lim = red[33];
        if (!isfinite(bvf) ? s > 0 : (bvf <= lim || bvf <= 0.f)) {
            rkeep = s;
            break;
        }
        if (bi != s) {
            df *cs = A + (size_t) s * lda, *cb = A + (size_t) bi * lda;
            for (int i = tm.tid; i < mrows; i += tm.nth) {
                const df t = cs[i];
                cs[i] = cb[i];
                cb[i] = t;
            }
            if (tm.tid == 0) {
                const df t = nrm[s];
                nrm[s] = nrm[bi];
                nrm[bi] = t;
                const df tr = nref[s];
                nref[s] = nref[bi];
                nref[bi] = tr;
                const int ti = pvt[s];
                pvt[s] = pvt[bi];
                pvt[bi] = ti;
            }
        }
        tm.sync();
        // Householder vector of column s (rows s..mrows-1), dlarfg convention, by the first warp.
        df *x = A + (size_t) s * lda;
        df *rts = reinterpret_cast<df *>(red + 40);  // tau and scale
        df t = df_f(0.f);
        if (warp == 0) {
            for (int i = s + 1 + lane; i < mrows; i += 32) t = df_fma(x[i], x[i], t);
            t = group_sum(t, 32);
        }
        if (tm.tid == 0) {
            const df alpha = x[s];
            df tau = df_f(0.f), scale = df_f(0.f), beta = alpha;
            if (t.h != 0.f) {
                const df nrmx = df_sqrt(df_fma(alpha, alpha, t));
                beta = alpha.h >= 0.f ? -nrmx : nrmx;
                tau = df_div(df_add(beta, -alpha), beta);
                scale = df_div(df_f(1.f), df_add(alpha, -beta));
            }
            x[s] = beta;
            rts[0] = tau;
            rts[1] = scale;
        }
        tm.sync();
        const df tau = rts[0], scale = rts[1];
        for (int i = s + 1 + tm.tid; i < mrows; i += tm.nth) x[i] = df_mul(x[i], scale);
        tm.sync();
        if (mrows <= 64) qrcp_apply_df<4>(tm, A, lda, mrows, ncols, s, x, tau, nrm, nref);
        else if (mrows <= 256) qrcp_apply_df<8>(tm, A, lda, mrows, ncols, s, x, tau, nrm, nref);
        else qrcp_apply_df<16>(tm, A, lda, mrows, ncols, s, x, tau, nrm, nref);
        tm.sync();
    }
    return rkeep;
}

// Shared variables of a team (of a cluster: in its first CTA).
struct CoreShared {
    int rot, rank, emax, cosine, tangent;
    double amax;
};

template <int RPL, class TM>
__device__ void core_update(const TM &tm, const DevUpdate *ups, const Workspace &ws, const Params &p, int slot,
                            double *sm, double *pool, int pool_doubles, CoreShared &sh);

// Doubles of the auxiliary arrays of an update of stack width k at the start of its team's shared memory.
__device__ __forceinline__ int core_aux_doubles(const Workspace &ws, int slot) {
    const int k = ws.meta[(size_t) slot * META_INTS + META_K];
    return 6 * (k > 0 ? k : 1) + SVD_AUX_FIXED;
}

// CTA of SVD_THREADS threads, in one of three team layouts chosen by the update's stack width k: heavy (k > k_heavy:
// more than half of the shared memory, the preconditioner's columns included: 115 to 166) — the whole CTA; light
// (kthr4 < k <= k_heavy) — two half-CTA teams of SVD_THREADS / 2 threads, one update each, each with half
// of the shared memory and its own named barrier; small (k <= kthr4: the core fits a quarter) — four teams
// of SVD_THREADS / 4 threads.  Small cores are latency-bound (per-step barriers, dependent FP64 chains), so
// four of them per SM hide each other's latency.  Wider updates are core_wide_kernel's.  With ws.order
// (sorted by decreasing k) the classes are contiguous: after the wide updates, a CTA takes a heavy one each, the
// next ceil(L / 2) take the L light updates in pairs, the rest the small ones in fours.  Without an order
// (one update per CTA) the team size follows the same class rule, so an update's arithmetic never
// depends on the launch it is part of.
template <int RPL>
__device__ void core_svd_cta(const DevUpdate *ups, int nup, const Workspace &ws, const Params &p, int team_doubles, int kthr4) {
    extern __shared__ __align__(16) double smem_all[];  // read as float4 at even offsets
    __shared__ CoreShared s_sh[4];
    __shared__ int s_end[3];  // first index behind the wide, heavy and light updates
    if (threadIdx.x < 3)
        s_end[threadIdx.x] = !ws.order ? 0 : (threadIdx.x == 0 ? ws.wide_updates(nup)
                                                               : ws.count_above(nup, threadIdx.x == 1 ? ws.k_heavy : kthr4));
    __syncthreads();
    constexpr int HALF = SVD_THREADS / 2, QUART = SVD_THREADS / 4;
    int idx, part = 0, teams;
    if (!ws.order) {
        idx = blockIdx.x;
        if (idx >= nup) return;
        const int key = ws.key(idx);
        if (key > ws.k_heavy) return;  // single updates: heavy ones on a cluster
        teams = key > kthr4 ? 2 : 4;
        if ((int) threadIdx.x >= SVD_THREADS / teams) return;
    } else {
        const int b = blockIdx.x, nh = s_end[1] - s_end[0], nl = s_end[2] - s_end[1], nlb = (nl + 1) / 2;
        teams = b < nh ? 1 : (b < nh + nlb ? 2 : 4);
        part = threadIdx.x / (SVD_THREADS / teams);
        if (teams == 1) {
            idx = s_end[0] + b;
        } else if (teams == 2) {
            idx = s_end[1] + 2 * (b - nh) + part;
            if (idx >= s_end[2]) return;  // the odd light update's partner slot stays idle
        } else {
            idx = s_end[2] + 4 * (b - nh - nlb) + part;
        }
    }
    if (idx >= nup) return;
    const int slot = ws.heavy(idx), doubles = 2 * team_doubles / teams;
    double *sm = smem_all + (size_t) part * doubles;
    const int aux = core_aux_doubles(ws, slot), tid = threadIdx.x % (SVD_THREADS / teams);
    if (teams == 1)
        core_update<RPL>(Team<SVD_THREADS>{tid, 1}, ups, ws, p, slot, sm, sm + aux, doubles - aux, s_sh[0]);
    else if (teams == 2)
        core_update<RPL>(Team<HALF>{tid, 1 + part}, ups, ws, p, slot, sm, sm + aux, doubles - aux, s_sh[part]);
    else
        core_update<RPL>(Team<QUART>{tid, 1 + part}, ups, ws, p, slot, sm, sm + aux, doubles - aux, s_sh[part]);
}

template <int RPL>
__global__ void __launch_bounds__(SVD_THREADS, 1) core_svd_kernel(const DevUpdate *ups, int nup, Workspace ws,
                                                               Params p, int team_doubles, int kthr4) {
    core_svd_cta<RPL>(ups, nup, ws, p, team_doubles, kthr4);
    wait_for_previous_launch();
}

// The wide updates (Workspace::wide_updates): a cluster of WIDE_CTAS
// CTAs each, the matrices in global memory (L2), the auxiliary arrays and shared variables in the first
// CTA's shared memory.  One SM's FP64 pipe took 35 ms for the Jacobi sweeps of a 200-column core and 180 ms for
// a 340-column one, and a chain of such updates bounds a multiply, however few they are.
template <int RPL>
__global__ void __cluster_dims__(WIDE_CTAS, 1, 1) __launch_bounds__(SVD_THREADS, 1)
    core_wide_kernel(const DevUpdate *ups, int nup, Workspace ws, Params p, int smem_doubles) {
    extern __shared__ __align__(16) double smem_all[];  // read as float4 at even offsets
    __shared__ CoreShared s_sh;
    __shared__ int s_wide;
    let_next_launch_start();
    const int rank = cluster_rank();
    const ClusterTeam<SVD_THREADS, WIDE_CTAS> tm{rank * SVD_THREADS + (int) threadIdx.x, rank};
    if (threadIdx.x == 0) s_wide = ws.order ? ws.wide_updates(nup) : nup;
    __syncthreads();
    const int H = s_wide, ncl = gridDim.x / WIDE_CTAS;
    double *sm = cluster_map(smem_all, 0);
    CoreShared &sh = *cluster_map(&s_sh, 0);
    for (int h = blockIdx.x / WIDE_CTAS; h < H; h += ncl) {
        const int slot = ws.heavy(h);
        if (ws.key(slot) <= ws.k_heavy) continue;
        const int aux = (core_aux_doubles(ws, slot) + 1) & ~1;
        tm.sync();  // the first CTA's shared memory is the previous update's no more (and exists)
        core_update<RPL>(tm, ups, ws, p, slot, sm, smem_all + aux, smem_doubles - aux, sh);
    }
    if ((int) (blockIdx.x / WIDE_CTAS) < H) tm.sync();  // no CTA leaves while another reads its shared memory
}

// Exponent of the largest entry of X (rows x cols), within +-1000 so that 2^e and 2^-e are normal (0 for a zero X).
template <class TM>
__device__ int core_exponent(const TM &tm, const double *X, int ldx, int rows, int cols, int *s_emax) {
    if (tm.tid == 0) *s_emax = 0;
    tm.sync();
    int em = 0;
    for (int j = tm.warp(); j < cols; j += tm.nw())
        for (int r = threadIdx.x & 31; r < rows; r += 32) {
            const int f = (int) ((__double_as_longlong(X[r + (size_t) j * ldx]) >> 52) & 0x7ff);
            em = em > f ? em : f;
        }
    for (int o = 16; o > 0; o >>= 1) {
        const int f = __shfl_xor_sync(0xffffffffu, em, o);
        em = em > f ? em : f;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(s_emax, em);
    tm.sync();
    const int e = *s_emax ? *s_emax - 1023 : 0;
    return e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
}

// X (rows x cols) <- X 2^e.
template <class TM>
__device__ void scale_columns(const TM &tm, double *X, int ldx, int rows, int cols, int e) {
    const double f = __hiloint2double((1023 + e) << 20, 0);
    for (int j = tm.warp(); j < cols; j += tm.nw())
        for (int r = threadIdx.x & 31; r < rows; r += 32) X[r + (size_t) j * ldx] *= f;
    tm.sync();
}

// The recompression core of one update (slot) by one team: auxiliary arrays at sm, `pool_doubles` of shared
// memory at pool (a cluster: of every CTA's own).
template <int RPL, class TM>
__device__ void core_update(const TM &tm, const DevUpdate *ups, const Workspace &ws, const Params &p, int slot,
                            double *sm, double *pool, int pool_doubles, CoreShared &sh) {
    int &s_rot = sh.rot, &s_rank = sh.rank, &s_emax = sh.emax;
    double &s_amax = sh.amax;
    constexpr bool CLUSTER = TM::ctas > 1;
    int *meta = ws.meta + (size_t) slot * META_INTS;
    if (meta[META_STATUS] != HCGB_OK || !meta[META_CKIND]) return;
    const int warp = tm.warp(), lane = threadIdx.x & 31, nw = tm.nw();
    const int lr = lane >> 2, lc = lane & 3;
    const int k = meta[META_K], m = meta[META_M], n = meta[META_N];
    const int kU = m < k ? m : k, kV = n < k ? n : k;
    const int ld = ws.ld, ldm = ws.kmax;
    double *base = ws.slot(slot);
    const double *RU = base + ws.off_ustack;
    const double *RV = base + ws.off_vstack;
    double *Mc = base + ws.off_mcopy;
    // Aux arrays at the start of the team's shared memory, sized by this update's stack width ka
    // (every index below is < k): sorted sigma, scratch, column norms, the sort permutation, the QR
    // pivots, the Jacobi scales and a reduction area (64 doubles + 128 ints).
    const int ka = k > 0 ? k : 1;
    double *sig = sm;
    double *inv = sig + ka;
    double *nrm = inv + ka;
    int *perm = reinterpret_cast<int *>(nrm + ka);
    int *pvt = perm + ka;
    double *dsc = nrm + ka + ka + 1;  // Jacobi column scales d and 1/d (2 ka)
    double *red = dsc + 2 * ka;
    int *redi = reinterpret_cast<int *>(red + SVD_RED_DOUBLES);
    // Working copy of M: shared memory when it fits, else the workspace.
    double *Mw;
    int ldw;
    if (!CLUSTER && (long) kU * kV <= (long) pool_doubles) {
        Mw = pool;
        ldw = kU;
    } else {
        Mw = base + ws.off_m;
        ldw = ldm;
    }

    // A cluster holds the columns of M in its CTAs' shared memory during the pivoted QR, as far as they fit (the working
    // copy takes the others).
    constexpr bool spread = CLUSTER;

    const long long t0 = clock64();
    // 1. M = R_U R_V^T on DMMA (R_U = triu of the U stack's top kU rows, likewise R_V), or the tile itself.
    if (ups[slot].direct) {
        const double *D = ups[slot].a.data;
        for (int j = warp; j < kV; j += nw)
            for (int i = lane; i < kU; i += 32) {
                const double v = D[i + (size_t) j * m];
                if (!spread) Mw[i + (size_t) j * ldw] = v;
                Mc[i + (size_t) j * ldm] = v;
            }
    } else {
        const int ntr = (kU + 7) >> 3, ntc = (kV + 7) >> 3;
        for (int idx = warp; idx < ntr * ntc; idx += nw) {
            const int tr = idx % ntr, tc = idx / ntr;
            const int i = tr * 8 + lr, j = tc * 8 + lr;
            double d0 = 0.0, d1 = 0.0;
            const int l0 = ((tr > tc ? tr : tc) * 8) & ~3;
            for (int l4 = l0; l4 < k; l4 += 4) {
                const int l = l4 + lc;
                const double av = (i < kU && l < k && l >= i) ? RU[i + (size_t) l * ld] : 0.0;
                const double bv = (j < kV && l < k && l >= j) ? RV[j + (size_t) l * ld] : 0.0;
                dmma(d0, d1, av, bv);
            }
            const int col = tc * 8 + 2 * lc;
            if (i < kU && col < kV) {
                if (!spread) Mw[i + (size_t) col * ldw] = d0;
                Mc[i + (size_t) col * ldm] = d0;
            }
            if (i < kU && col + 1 < kV) {
                if (!spread) Mw[i + (size_t) (col + 1) * ldw] = d1;
                Mc[i + (size_t) (col + 1) * ldm] = d1;
            }
        }
    }
    tm.sync();

    // 2. Rank-revealing QR with column pivoting, M P = Q R, stopped once every remaining column
    //    is below QRCP_STOP (1e-2) of the truncation threshold.  The dropped block R22 lies far
    //    below the threshold: it cannot carry a kept singular value, it moves the kept ones by at
    //    most ||R22||_2 <= sqrt(kV) * 1e-2 * threshold (in practice ~1e-6 relative), and it only
    //    holds directions the truncation discards anyway.  The Jacobi stage then works on the
    //    rk rows above it.  (Fixed-rank mode keeps every row.)
    constexpr double QRCP_STOP = 1e-2;
    double stop2 = -1.0, rel = 0.0;
    if (p.fixed_rank <= 0) {
        if (p.truncated) {
            stop2 = 0.0;
            rel = QRCP_STOP * p.accuracy;  // |r_00| <= sigma_0, so this threshold is conservative
        } else {
            stop2 = (QRCP_STOP * p.accuracy) * (QRCP_STOP * p.accuracy);
        }
    }
    const long long t1 = clock64();
    int rk = 0;
    double *XV = base + ws.off_xv;
    double up = 1.0;  // mixed form: Mw holds float-float values of M / up from here to step 3
    const bool ff = TM::nth < SVD_THREADS && p.mode == 1;  // heavy and wide cores are FP64 in every form
    if (ff) {
        // Exact power-of-two scaling that brings the largest entry of M near 1 (float range), then
        // the pivoted QR and the Jacobi sweeps in float-float arithmetic on the FP32 pipe.
        if (tm.tid == 0) s_emax = 0;
        tm.sync();
        int em = 0;
        for (int e = tm.tid; e < kU * kV; e += tm.nth) {
            const int ef = (int) ((__double_as_longlong(Mw[(e % kU) + (size_t) (e / kU) * ldw]) >> 52) & 0x7ff);
            em = em > ef ? em : ef;
        }
        atomicMax(&s_emax, em);
        tm.sync();
        const int eshift = s_emax ? s_emax - 1023 : 0;
        up = __hiloint2double((1023 + eshift) << 20, 0);
        const double down = __hiloint2double((1023 - eshift) << 20, 0);
        df *Md = reinterpret_cast<df *>(Mw);
        for (int e = tm.tid; e < kU * kV; e += tm.nth) {
            const size_t o = (e % kU) + (size_t) (e / kU) * ldw;
            Md[o] = df(Mw[o] * down);
        }
        tm.sync();
        const float stop2f = stop2 > 0.0 ? (float) (stop2 * down * down) : (float) stop2;
        rk = qrcp_truncated_df(tm, Md, ldw, kU, kV, stop2f, (float) (rel * rel), reinterpret_cast<df *>(nrm),
                               reinterpret_cast<df *>(inv), pvt, reinterpret_cast<float *>(red), redi);
    } else if (spread) {
        if constexpr (CLUSTER) {  // lanes per column as in qrcp_truncated
            rk = kU <= 64    ? qrcp_cluster<4>(tm, Mc, ldm, kU, kV, stop2, rel, XV, ld, pvt, pool, pool_doubles, Mw, ldw)
                 : kU <= 256 ? qrcp_cluster<8>(tm, Mc, ldm, kU, kV, stop2, rel, XV, ld, pvt, pool, pool_doubles, Mw, ldw)
                             : qrcp_cluster<16>(tm, Mc, ldm, kU, kV, stop2, rel, XV, ld, pvt, pool, pool_doubles, Mw, ldw);
        }
    } else {
        rk = qrcp_truncated(tm, Mw, ldw, kU, kV, stop2, rel, nrm, inv, pvt, red, redi);
    }
    const long long t2 = clock64();
    if (rk < 1) rk = 1;
    // 3. X = R(0:rk, :)^T (kV x rk) in XV.
    for (int i = spread ? rk : warp; i < rk; i += nw)
        for (int l = lane; l < kV; l += 32) {
            double x = 0.0;
            if (l >= i) {
                const double *e = Mw + i + (size_t) (ff ? l : pvt[l]) * ldw;  // the float-float QR swaps columns
                x = ff ? (double) *reinterpret_cast<const df *>(e) * up : *e;
            }
            XV[l + (size_t) i * ld] = x;
        }
    tm.sync();
    double *X = Mw;
    const int ldx = kV;
    // 4. One-sided Jacobi on the rk columns of X: X J = W with orthogonal columns: sigma_i = ||w_i||, right
    //    singular vectors P W Sigma^-1.  Preconditioned in single precision from precond_min columns on
    //    (where its buffers fit); what that leaves, and smaller cores, go to the FP64 sweeps.
    int sweeps = 0;
    bool converged = true;
    const double tol64 = 8.0 * DBL_EPSILON * (double) (kV > 1 ? kV : 1);
    const double *Xs = XV;
    int lds = ld;
    if (rk >= p.precond_min && rk >= 4) {
        PrecondBuffers b;
        const int x4 = (kV + 3) >> 2, j4 = (rk + 3) >> 2;
        bool fits;
        if constexpr (CLUSTER) {
            b.ls4 = x4 + j4;
            b.blocks = SWEEP_BLOCKS;
            b.g8 = false;
            b.y = reinterpret_cast<float4 *>(base + ws.off_mixed);
            b.buf = reinterpret_cast<float4 *>(pool);
            b.buf_quads = pool_doubles / 2;
            b.wh = reinterpret_cast<df *>(XV);
            b.ldh = ld;
            b.v = reinterpret_cast<float *>(b.y);
            b.ldv = 4 * b.ls4;
            fits = 4 * (size_t) b.ls4 * rk <= ws.mixed_floats && 2 * b.ls4 <= b.buf_quads;
        } else {
            b.ls4 = precond_quads(x4, j4);
            b.blocks = k > ws.k_heavy ? SWEEP_BLOCKS : 0;  // as on a cluster
            b.g8 = rk <= (k <= SMALL_K ? 32 : 64);
            const int skip = (int) ((reinterpret_cast<uintptr_t>(pool) >> 3) & 1);
            b.y = reinterpret_cast<float4 *>(pool + skip);
            b.buf = nullptr;
            b.buf_quads = 0;
            b.wh = reinterpret_cast<df *>(pool);
            b.ldh = (long) (kV | 1) * rk <= (long) pool_doubles ? (kV | 1) : kV;
            b.v = reinterpret_cast<float *>(base + ws.off_mixed);
            b.ldv = rk;
            fits = Mw == pool && 2L * b.ls4 * rk + skip <= (long) pool_doubles;
        }
        b.e64 = base + ws.off_m;
        b.w = base + ws.off_mixed;
        if constexpr (!CLUSTER) {
            // E, W and V in shared memory behind y / wh, as far as they fit
            const long ly = 2L * b.ls4 * rk + 1, lh = (long) b.ldh * rk;
            long top = ly > lh ? ly : lh;
            auto place = [&](long doubles) -> double * {
                if (top + doubles > (long) pool_doubles) return nullptr;
                double *at = pool + top;
                top += doubles;
                return at;
            };
            if (double *at = place((long) rk * rk)) b.e64 = at;
            if (double *at = place((long) kV * rk)) b.w = at;
            if (double *at = place(((long) rk * rk + 1) / 2)) b.v = reinterpret_cast<float *>(at);
        }
        if (fits && jacobi_precond(tm, XV, ld, kV, rk, b, reinterpret_cast<df *>(nrm), perm, &s_rot, &s_emax,
                                   &sh.cosine, &sh.tangent, (float) tol64, &sweeps, &converged)) {
            Xs = b.w;
            lds = kV;
            if (converged) sweeps = -sweeps;
        }
    }
    tm.sync();
    for (int i = warp; i < rk; i += nw)
        for (int l = lane; l < kV; l += 32) X[l + (size_t) i * ldx] = Xs[l + (size_t) i * lds];
    tm.sync();
    if (sweeps < 0) {
        sweeps = -sweeps;  // the corrections left orthogonal columns
    } else {
        int more = 0;
        // The sweeps' tests multiply squared norms with one another: columns far from 1 (a^2 below ~1e-300 or above
        // 1e300, with the factors tol^2 and noise^2 between them) are scaled by an exact power of two for them.
        const int e = core_exponent(tm, X, ldx, kV, rk, &s_emax);
        const bool scaled = e < -150 || e > 150;
        if (scaled) scale_columns(tm, X, ldx, kV, rk, -e);
        // on a cluster, a core that one SM could hold takes that SM's lanes per pair
        jacobi_dispatch<RPL>(tm, X, ldx, kV, rk, nrm, &s_rot, &s_amax, &more, &converged, tol64, MAX_JACOBI_SWEEPS, dsc,
                             ka, CLUSTER ? k <= ws.k_wide : Mw == pool);
        if (scaled) scale_columns(tm, X, ldx, kV, rk, e);
        sweeps += more;
    }

    const long long t3 = clock64();
    // 5. Singular values, descending order (stable), rank rule (omp/kernels.cpp:82-104).
    for (int j = warp; j < rk; j += nw) {
        const double *col = X + (size_t) j * ldx;
        double t = 0.0;
        for (int r = lane; r < kV; r += 32) t = fma(col[r], col[r], t);
        t = warp_sum(t);
        // unsorted sigma, temporarily in inv[]; -1 for a NaN, so that the order below is total and perm a
        // permutation whatever the columns hold
        if (lane == 0) inv[j] = t >= 0.0 ? sqrt(t) : -1.0;
    }
    tm.sync();
    for (int j = tm.tid; j < rk; j += tm.nth) {
        const double sj = inv[j];
        int pos = 0;
        for (int l = 0; l < rk; l++) {
            const double sl = inv[l];
            pos += (sl > sj) || (sl == sj && l < j);
        }
        perm[pos] = j;
        sig[pos] = sj < 0.0 ? __longlong_as_double(NRM_SIGN_MASK) : sj;
    }
    tm.sync();
    if (tm.tid == 0) {
        const int sizeS = kU < kV ? kU : kV;
        int r;
        if (p.fixed_rank > 0) {
            r = p.fixed_rank < k ? p.fixed_rank : k;
        } else {
            // sigma_i for i >= rk are below the threshold by construction of the QR stop.
            r = rk < sizeS ? rk : sizeS;
            const double thr = p.truncated ? p.accuracy * sig[0] : p.accuracy;
            for (int i = 1; i < rk; i++)
                if (sig[i] < thr) {
                    r = i;
                    break;
                }
        }
        if (r < 1) r = 1;
        const int maxr = ups[slot].c.max_rank;
        if (r > maxr) r = maxr;
        if (r > rk) r = rk;
        s_rank = r;
        base[ws.off_sigma] = sig[0];  // the largest singular value (the learned form's residual test)
        meta[META_NEWRANK] = r;
        meta[META_SWEEPS] = sweeps;
        meta[META_CORE_COLS] = rk;
        if (!converged) meta[META_STATUS] = HCGB_NOT_CONVERGED;
    }
    tm.sync();
    const int r = s_rank;
    for (int i = tm.tid; i < r; i += tm.nth) inv[i] = sig[i] > 1e-150 ? 1.0 / (sig[i] * sig[i]) : 0.0;

    // 6. Right factor in the small basis: XV = P W_r (= V_r Sigma_r), n rows, zero below kV.
    for (int i = warp; i < r; i += nw) {
        const double *w = X + (size_t) perm[i] * ldx;
        for (int l = lane; l < kV; l += 32) XV[pvt[l] + (size_t) i * ld] = w[l];
        for (int l = kV + lane; l < n; l += 32) XV[l + (size_t) i * ld] = 0.0;
    }
    tm.sync();

    // 7. Left factor in the small basis: C.U[:, i] = [M XV[:, i] / sigma_i^2 ; 0] (= U_r), on DMMA.
    double *CU = ups[slot].c.data;
    const int ldcu = ups[slot].c.rows;
    {
        const int ntr = (kU + 7) >> 3, ntc = (r + 7) >> 3;
        for (int idx = warp; idx < ntr * ntc; idx += nw) {
            const int tr = idx % ntr, tc = idx / ntr;
            const int irow = tr * 8 + lr, icol = tc * 8 + lr;
            const double *vcol = XV + (size_t) (icol < r ? icol : 0) * ld;
            double d0 = 0.0, d1 = 0.0;
            for (int l4 = 0; l4 < kV; l4 += 4) {
                const int l = l4 + lc;
                const double av = (irow < kU && l < kV) ? Mc[irow + (size_t) l * ldm] : 0.0;
                const double bv = (icol < r && l < kV) ? vcol[l] : 0.0;
                dmma(d0, d1, av, bv);
            }
            const int col = tc * 8 + 2 * lc;
            if (irow < kU && col < r) CU[irow + (size_t) col * ldcu] = d0 * inv[col];
            if (irow < kU && col + 1 < r) CU[irow + (size_t) (col + 1) * ldcu] = d1 * inv[col + 1];
        }
        for (int i = warp; i < r; i += nw)
            for (int l = kU + lane; l < m; l += 32) CU[l + (size_t) i * ldcu] = 0.0;
    }
    if (tm.tid == 0) {
        const long long t4 = clock64();
        meta[META_KC_PRODUCT] = (int) ((t1 - t0) >> 10);
        meta[META_KC_QRCP] = (int) ((t2 - t1) >> 10);
        meta[META_KC_JACOBI] = (int) ((t3 - t2) >> 10);
        meta[META_KC_FACTORS] = (int) ((t4 - t3) >> 10);
    }
}

}  // namespace

namespace {

// Half of the per-block opt-in limit of shared memory (less a reserve for the kernel's static shared variables), in
// doubles.
long svd_half_sm_doubles() {
    static const int optin = [] {  // thread-safe one-time initialisation
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        return v > 0 ? v : 48 * 1024;
    }();
    return (optin - 256) / 2 / (long) sizeof(double);
}

// Doubles a core of k columns takes: its aux arrays, the k x k working copy and the preconditioner's padded columns (one
// double aligns them).
long core_doubles(long k) {
    const long q = (k + 3) / 4;
    return 6 * k + SVD_AUX_FIXED + std::max(k * k, 2L * precond_quads((int) q, (int) q) * k + 1);
}

int widest_core(long doubles) {
    int k = 0;
    while (core_doubles(k + 1) <= doubles) k++;
    return k;
}

// Doubles of shared memory per half-CTA team: what a core of kmax columns takes, capped at half of an SM's, and never
// below the aux arrays.
int svd_team_doubles(int kmax) {
    const long aux = 6L * kmax + SVD_AUX_FIXED, cap = svd_half_sm_doubles();
    const long want = std::max(aux + (long) kmax * kmax + 14L * kmax, core_doubles(kmax));
    long t = want < cap ? want : cap;
    if (t < aux) t = aux;  // checked against the device limit by the caller
    return (int) t;
}

}  // namespace

size_t svd_smem_bytes(int kmax) { return 2 * sizeof(double) * (size_t) svd_team_doubles(kmax); }

// Register tiles of the FP64 sweeps: up to 16 rows a lane (longer columns take the looped sweep).
constexpr int CORE_RPL = 16;

// Widths up to which a core fits its team (one that the preconditioner's columns did not fit would fall back to the FP64
// sweeps, twice the time at 25 columns).  A whole and half an SM decide the order of the sweeps and the form of the
// pivoted QR, so they follow from the SM alone and not from the capacities of a launch's tiles; a quarter only decides
// which team takes the core.  A 110-column core of width 128 takes a cluster of eight 4,300 kcycles and one SM
// alone 7,900: heavy ones go to clusters only while SMs are idle, wide ones always.
void core_classes(int kmax, int *whole, int *half, int *quarter) {
    *whole = widest_core(2 * svd_half_sm_doubles());
    *half = widest_core(svd_half_sm_doubles());
    *quarter = widest_core(svd_team_doubles(kmax) / 2);
}

void set_core_classes(Workspace *ws) {
    int quarter;
    core_classes(ws->kmax, &ws->k_wide, &ws->k_heavy, &quarter);
}

static void launch_core_wide(const DevUpdate *ups, int n, Workspace ws, Params p, cudaStream_t st) {
    const int aux = 6 * ws.kmax + SVD_AUX_FIXED + 1;
    // a pair of column blocks, or (wider cores) as many columns as there is room for
    const int most = 2 * svd_team_doubles(ws.kmax);
    const int doubles = ws.kmax <= WIDE_POOL_K ? std::min(aux + WIDE_POOL_DOUBLES, most) : most;
    const size_t bytes = sizeof(double) * (size_t) doubles;
    cudaFuncSetAttribute(core_wide_kernel<CORE_RPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes);
    const int ctas = std::min(n, WIDE_CLUSTERS) * WIDE_CTAS;
    { core_wide_kernel<CORE_RPL><<<ctas, SVD_THREADS, bytes, st>>>(ups, n, ws, p, doubles); note_launch(); }
}

void launch_core_svd(const DevUpdate *ups, int n, Workspace ws, Params p, cudaStream_t st) {
    const int team = svd_team_doubles(ws.kmax);
    const size_t smem = 2 * sizeof(double) * (size_t) team;
    int whole, half, quarter;
    core_classes(ws.kmax, &whole, &half, &quarter);
    cudaFuncSetAttribute(core_svd_kernel<CORE_RPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    const bool wide = ws.kmax > ws.k_heavy;
    if (wide) launch_core_wide(ups, n, ws, p, st);
    launch_beside(wide, 1, n, SVD_THREADS, smem, st, core_svd_kernel<CORE_RPL>, ups, n, ws, p, team, quarter);
}

}  // namespace hcgb
