// Dense per-tile building blocks of a tile Cholesky: potrf, trsm, syrk (FP64).
//
// Replace HCoreKernels<T>::potrf / trsm / syrk on the GPU (src/kernels/cuda/kernels.cpp:290-306,
// src/kernels/cuda/CudaKernels.cu:1019-1049: cuSOLVER Xpotrf, cuBLAS trsm/syrk) with the
// semantics of LAPACK dpotrf and BLAS dtrsm / dsyrk (column-major), which the CPU backend calls
// (src/kernels/omp/kernels.cpp:234-282).
#include "internal.cuh"

namespace hcgb {

namespace {

constexpr int CT = 1024;

// Blocked right-looking Cholesky.  One launch per 32-column block solves the rows below it, one updates the
// trailing 32 x 32 tiles over the whole GPU; the CTA of the next diagonal tile factors it on the spot, so a
// block costs two launches.  (One CTA walked the columns, each a left-looking product from L2, bound by one
// SM's FP64 pipe and dependent loads: with the panel solve below, five tiles of 512 and ten panel tiles took 285 ms
// of a tile Cholesky, 10 ms now.)  L(i, k) stands at A[i rs + k cs]: lower triangle
// rs = 1, cs = lda, upper the other way round.  Every L(i, j) takes its products in ascending k.
// A launch acts on failures of earlier launches alone (*info at most the last column it depends on), so that
// all its threads decide alike whenever they read the word that one of its own CTAs may write.
constexpr int PB = 32;

// Factors the leading nb x nb block held in shared memory (lower part); returns the failing column + 1 or 0.
__device__ int potrf_block(double (*T)[PB + 1], int nb) {
    for (int j = 0; j < nb; j++) {
        const double d = T[j][j];
        if (!(d > 0.0)) return j + 1;
        const double ljj = sqrt(d);
        __syncthreads();
        if (threadIdx.x == 0) T[j][j] = ljj;
        for (int i = j + 1 + (int) threadIdx.x; i < nb; i += blockDim.x) T[i][j] /= ljj;
        __syncthreads();
        for (int e = threadIdx.x; e < (nb - 1 - j) * PB; e += blockDim.x) {
            const int i = j + 1 + e / PB, k = e % PB;
            if (k > j && k <= i) T[i][k] = fma(-T[i][j], T[k][j], T[i][k]);
        }
        __syncthreads();
    }
    return 0;
}

__global__ void __launch_bounds__(256) potrf_first_kernel(double *A, int n, int rs, int cs, int *info) {
    __shared__ double T[PB][PB + 1];
    const int nb = n < PB ? n : PB;
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
        const int i = e % nb, k = e / nb;
        if (i >= k) T[i][k] = A[(size_t) i * rs + (size_t) k * cs];
    }
    __syncthreads();
    const int bad = potrf_block(T, nb);
    __syncthreads();
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
        const int i = e % nb, k = e / nb;
        if (i >= k) A[(size_t) i * rs + (size_t) k * cs] = T[i][k];
    }
    if (threadIdx.x == 0) *info = bad;
}

// Rows below block column j0 (width PB; the columns before a failing one): 32 rows a CTA, four threads a row, each with
// every fourth column.
__global__ void __launch_bounds__(128) potrf_panel_kernel(double *A, int n, int j0, int rs, int cs, const int *info) {
    __shared__ double D[PB][PB + 1];
    const int bad = *info, cols = bad ? bad - 1 - j0 : PB;
    if (cols <= 0) return;
    for (int e = threadIdx.x; e < PB * PB; e += blockDim.x) {
        const int i = e % PB, k = e / PB;
        D[i][k] = i >= k ? A[(size_t) (j0 + i) * rs + (size_t) (j0 + k) * cs] : 0.0;
    }
    __syncthreads();
    const int row = j0 + PB + blockIdx.x * 32 + (threadIdx.x >> 2), q = threadIdx.x & 3;
    const bool in = row < n;
    double *r = A + (size_t) (in ? row : 0) * rs + (size_t) j0 * cs;
    double t[PB / 4];
#pragma unroll
    for (int u = 0; u < PB / 4; u++) t[u] = in ? r[(size_t) (4 * u + q) * cs] : 0.0;
#pragma unroll
    for (int j = 0; j < PB; j++) {
        double x = t[j / 4] / D[j][j];
        x = __shfl_sync(0xffffffffu, x, j & 3, 4);
        if (q == (j & 3)) t[j / 4] = x;
#pragma unroll
        for (int u = 0; u < PB / 4; u++) {
            const int k = 4 * u + q;
            if (4 * u + 3 > j && k > j) t[u] = fma(-x, D[k][j], t[u]);
        }
    }
    if (in)
#pragma unroll
        for (int u = 0; u < PB / 4; u++)
            if (4 * u + q < cols) r[(size_t) (4 * u + q) * cs] = t[u];
}

// Trailing tiles (ti, tj), ti >= tj, behind block column j0: A -= L_i L_j^T; tile (0, 0) is factored too.
__global__ void __launch_bounds__(256) potrf_update_kernel(double *A, int n, int j0, int rs, int cs, int *info) {
    __shared__ double Li[PB][PB + 1], Lj[PB][PB + 1];
    const int bad_before = *info;
    if (bad_before && bad_before <= j0 + PB) return;  // tile (0, 0) of this launch writes j0 + PB + 1 or more
    int ti = 0, base = 0;
    while (base + ti + 1 <= (int) blockIdx.x) {
        base += ti + 1;
        ti++;
    }
    const int tj = (int) blockIdx.x - base, i0 = j0 + PB * (1 + ti), k0 = j0 + PB * (1 + tj);
    const int ni = n - i0 < PB ? n - i0 : PB, nk = n - k0 < PB ? n - k0 : PB;
    for (int e = threadIdx.x; e < PB * PB; e += blockDim.x) {
        const int i = e % PB, l = e / PB;
        Li[i][l] = i < ni ? A[(size_t) (i0 + i) * rs + (size_t) (j0 + l) * cs] : 0.0;
        Lj[i][l] = i < nk ? A[(size_t) (k0 + i) * rs + (size_t) (j0 + l) * cs] : 0.0;
    }
    __syncthreads();
    const int x = threadIdx.x & 15, y = threadIdx.x >> 4;
    double t[2][2];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int i = x + 16 * u, k = y + 16 * v;
            t[u][v] = (i < ni && k < nk && i0 + i >= k0 + k) ? A[(size_t) (i0 + i) * rs + (size_t) (k0 + k) * cs] : 0.0;
        }
#pragma unroll 4
    for (int l = 0; l < PB; l++) {
        const double a0 = Li[x][l], a1 = Li[x + 16][l], b0 = Lj[y][l], b1 = Lj[y + 16][l];
        t[0][0] = fma(-a0, b0, t[0][0]);
        t[0][1] = fma(-a0, b1, t[0][1]);
        t[1][0] = fma(-a1, b0, t[1][0]);
        t[1][1] = fma(-a1, b1, t[1][1]);
    }
    const bool next = ti == 0;
    if (next) __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int i = x + 16 * u, k = y + 16 * v;
            if (i < ni && k < nk && i0 + i >= k0 + k) {
                if (next) Li[i][k] = t[u][v];
                else A[(size_t) (i0 + i) * rs + (size_t) (k0 + k) * cs] = t[u][v];
            }
        }
    if (!next) return;
    __syncthreads();
    const int bad = potrf_block(Li, ni);
    __syncthreads();
    for (int e = threadIdx.x; e < ni * ni; e += blockDim.x) {
        const int i = e % ni, k = e / ni;
        if (i >= k) A[(size_t) (i0 + i) * rs + (size_t) (i0 + k) * cs] = Li[i][k];
    }
    if (threadIdx.x == 0 && bad) *info = i0 + bad;
}

// Columns k >= from of the triangle (L(i, k), i >= k) copied between A (ld lda) and keep (ld n); a CTA a stored column.
__global__ void __launch_bounds__(256) potrf_copy_kernel(int uplo, int n, int from, const double *src, int lds, double *dst,
                                                         int ldd) {
    const int c = blockIdx.x, r0 = uplo == 0 ? c : from, r1 = uplo == 0 ? n : c + 1;
    if (uplo == 0 && c < from) return;
    for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) dst[r + (size_t) c * ldd] = src[r + (size_t) c * lds];
}

// op(A) X = alpha B (side 0) or X op(A) = alpha B (side 1); X overwrites B (m x n, ld ldb).
// Reduced to S y = alpha b for every vector b: columns of B with S = op(A) (side 0), or rows of B
// with S = op(A)^T (side 1); S is lower or upper triangular and solved by substitution, one
// step per row of S with all vectors updated in parallel.
__global__ void __launch_bounds__(CT) trsm_kernel(int side, int uplo, int trans, int diag, int m, int n, double alpha,
                                                  const double *A, int lda, double *B, int ldb) {
    const int len = side == 0 ? m : n;      // order of S
    const int count = side == 0 ? n : m;    // number of vectors
    // S(i, k): side 0: op(A)(i, k); side 1: op(A)(k, i).
    const bool t_eff = (side == 0) ? (trans != 0) : (trans == 0);
    const bool lower_s = (uplo == 0) != t_eff;
    auto S = [&](int i, int k) -> double { return t_eff ? A[k + (size_t) i * lda] : A[i + (size_t) k * lda]; };
    auto Bref = [&](int i, int v) -> double & { return side == 0 ? B[i + (size_t) v * ldb] : B[v + (size_t) i * ldb]; };
    for (int e = threadIdx.x; e < len * count; e += blockDim.x) Bref(e % len, e / len) *= alpha;
    __syncthreads();
    for (int step = 0; step < len; step++) {
        const int i = lower_s ? step : len - 1 - step;
        if (diag == 0) {
            const double sii = S(i, i);
            for (int v = threadIdx.x; v < count; v += blockDim.x) Bref(i, v) /= sii;
        }
        __syncthreads();
        // eliminate x_i from the remaining rows
        const int rest = lower_s ? len - 1 - i : i;
        for (int e = threadIdx.x; e < rest * count; e += blockDim.x) {
            const int r = e % rest, v = e / rest;
            const int k = lower_s ? i + 1 + r : r;
            Bref(k, v) = fma(-S(k, i), Bref(i, v), Bref(k, v));
        }
        __syncthreads();
    }
}

// C = alpha op(A) op(A)^T + beta C on the uplo triangle of C (n x n); op(A) is n x k.
__global__ void syrk_kernel(int uplo, int trans, int n, int k, double alpha, const double *A, int lda, double beta,
                            double *C, int ldc) {
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || j >= n) return;
    if (uplo == 0 ? (i < j) : (i > j)) return;
    double s = 0.0;
    for (int l = 0; l < k; l++) {
        const double a = trans ? A[l + (size_t) i * lda] : A[i + (size_t) l * lda];
        const double b = trans ? A[l + (size_t) j * lda] : A[j + (size_t) l * lda];
        s = fma(a, b, s);
    }
    double *c = C + i + (size_t) j * ldc;
    *c = alpha * s + (beta != 0.0 ? beta * *c : 0.0);
}

// Sets the strict uplo triangle of A (n x n, ld lda) to value (HCoreKernels::FillMatrixTriangle,
// src/kernels/omp/kernels.cpp:246-264).
__global__ void fill_triangle_kernel(int uplo, int n, double *A, int lda, double value) {
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || j >= n) return;
    if (uplo == 0 ? (i > j) : (i < j)) A[i + (size_t) j * lda] = value;
}

// Panel solve of a tile Cholesky step: for every compressed_vt tile of the panel, W <- L^-1 W
// (Left, Lower, NoTrans, NonUnit, alpha 1 on the W region, rows x rank, ld rows): HCore<T>::Trsm
// as the tile Cholesky applies it (src/api/HCore.cpp:623-647), the rank read on the device.  One CTA per
// tile and TRSM_COLS columns, which stay in shared memory: blocks of 32 rows are solved, then taken out of
// the rows below.  Every element takes the same operations in the same order as in trsm_kernel, so the
// results are identical.  (One CTA took a tile, one row a step through L2.)
constexpr int TRSM_COLS = 4, TRSM_THREADS = 256;
__global__ void __launch_bounds__(TRSM_THREADS) trsm_panel_kernel(const double *L, int nb, int ldl, const DevTile *tiles,
                                                                  int in_smem) {
    extern __shared__ double smem_w[];  // nb x TRSM_COLS, where that fits
    __shared__ double D[PB][PB + 1];
    const DevTile t = tiles[blockIdx.y];
    const int r = *t.rank, c0 = blockIdx.x * TRSM_COLS;
    if (r <= 0 || r > t.max_rank || t.rows != nb || c0 >= r) return;
    const int nc = r - c0 < TRSM_COLS ? r - c0 : TRSM_COLS;
    double *W = t.v + (size_t) c0 * nb;
    double *Ws = in_smem ? smem_w : W;
    if (in_smem)
        for (int e = threadIdx.x; e < nb * nc; e += TRSM_THREADS) Ws[e] = W[e];
    for (int i0 = 0; i0 < nb; i0 += PB) {
        const int ni = nb - i0 < PB ? nb - i0 : PB;
        __syncthreads();
        for (int e = threadIdx.x; e < ni * ni; e += TRSM_THREADS) {
            const int i = e % ni, k = e / ni;
            if (i >= k) D[i][k] = L[(i0 + i) + (size_t) (i0 + k) * ldl];
        }
        __syncthreads();
        if ((int) threadIdx.x < 32 * nc) {  // a warp per column, a lane per row
            const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
            double w = lane < ni ? Ws[i0 + lane + c * nb] : 0.0;
            for (int i = 0; i < ni; i++) {
                if (lane == i) w /= D[i][i];
                const double wi = __shfl_sync(0xffffffffu, w, i);
                if (lane > i && lane < ni) w = fma(-D[lane][i], wi, w);
            }
            if (lane < ni) Ws[i0 + lane + c * nb] = w;
        }
        __syncthreads();
        for (int k = i0 + ni + threadIdx.x; k < nb; k += TRSM_THREADS) {
            double w[TRSM_COLS];
#pragma unroll
            for (int c = 0; c < TRSM_COLS; c++) w[c] = c < nc ? Ws[k + c * nb] : 0.0;
#pragma unroll 8
            for (int i = 0; i < ni; i++) {
                const double l = -L[k + (size_t) (i0 + i) * ldl];
#pragma unroll
                for (int c = 0; c < TRSM_COLS; c++)
                    if (c < nc) w[c] = fma(l, Ws[i0 + i + c * nb], w[c]);
            }
#pragma unroll
            for (int c = 0; c < TRSM_COLS; c++)
                if (c < nc) Ws[k + c * nb] = w[c];
        }
    }
    __syncthreads();
    if (in_smem)
        for (int e = threadIdx.x; e < nb * nc; e += TRSM_THREADS) W[e] = Ws[e];
}

}  // namespace

void launch_trsm_panel(const double *L, int nb, int ldl, const DevTile *tiles, int count, int max_rank, cudaStream_t st) {
    if (count <= 0 || max_rank <= 0) return;
    size_t smem = sizeof(double) * (size_t) nb * TRSM_COLS;
    if (smem > 200 * 1024) smem = 0;
    cudaFuncSetAttribute(trsm_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    const dim3 grid((max_rank + TRSM_COLS - 1) / TRSM_COLS, count);
    { trsm_panel_kernel<<<grid, TRSM_THREADS, smem, st>>>(L, nb, ldl, tiles, smem > 0); note_launch(); }
}

void launch_fill_triangle(int uplo, int n, double *A, int lda, double value, cudaStream_t st) {
    dim3 blk(32, 8), grid((n + 31) / 32, (n + 7) / 8);
    { fill_triangle_kernel<<<grid, blk, 0, st>>>(uplo, n, A, lda, value); note_launch(); }
}

void launch_potrf_restore(double *A, int n, int lda, int uplo, int failed, const double *keep, cudaStream_t st) {
    { potrf_copy_kernel<<<n, 256, 0, st>>>(uplo, n, failed - 1, keep, n, A, lda); note_launch(); }
}

void launch_potrf(double *A, int n, int lda, int uplo, int *info_dev, double *keep, cudaStream_t st) {
    const int rs = uplo == 0 ? 1 : lda, cs = uplo == 0 ? lda : 1;
    if (keep) { potrf_copy_kernel<<<n, 256, 0, st>>>(uplo, n, 0, A, lda, keep, n); note_launch(); }
    { potrf_first_kernel<<<1, 256, 0, st>>>(A, n, rs, cs, info_dev); note_launch(); }
    for (int j0 = 0; j0 + PB < n; j0 += PB) {
        const int rest = (n - j0 - 1) / PB;  // row blocks below
        { potrf_panel_kernel<<<rest, 128, 0, st>>>(A, n, j0, rs, cs, info_dev); note_launch(); }
        { potrf_update_kernel<<<rest * (rest + 1) / 2, 256, 0, st>>>(A, n, j0, rs, cs, info_dev); note_launch(); }
    }
}

void launch_trsm(int side, int uplo, int trans, int diag, int m, int n, double alpha, const double *A, int lda,
                 double *B, int ldb, cudaStream_t st) {
    { trsm_kernel<<<1, CT, 0, st>>>(side, uplo, trans, diag, m, n, alpha, A, lda, B, ldb); note_launch(); }
}

void launch_syrk(int uplo, int trans, int n, int k, double alpha, const double *A, int lda, double beta, double *C,
                 int ldc, cudaStream_t st) {
    dim3 blk(16, 16), grid((n + 15) / 16, (n + 15) / 16);
    { syrk_kernel<<<grid, blk, 0, st>>>(uplo, trans, n, k, alpha, A, lda, beta, C, ldc); note_launch(); }
}

}  // namespace hcgb
