// Internal declarations shared by the CUDA translation units of libhcgb.
//
// Execution model of one batched call (a "wave" of independent tile updates, one
// update per C tile):
//   plan      : read the device-side ranks, choose the stacking side, and resolve
//               every factor product into a GemmJob (no host round trip)
//   stack     : copy/scale/transpose the C factors into the stacked bases
//               U = [Cu | alpha*Ua'] (m x k), V = [beta*Cv^T | Vb'] (n x k)
//   gemm x3   : the factor products, written straight into the stacks (or into a dense C):
//               a schedule kernel compacts the wave's output tiles, then persistent FP64 DMMA
//               (small) and FP64-accurate 16-bit tensor-core (large) product kernels
//   order     : updates sorted by stack width (the heavy stages' CTA order)
//   qr        : blocked Householder QR of both stacks (plain: panel SIMT + trailing DMMA;
//               mixed: float-float on the FP32 pipe)
//   core_svd  : M = R_U R_V^T, pivoted QR, one-sided Jacobi, rank truncation, new factors in
//               the small basis
//   apply_q   : new U = Q_U [U_r; 0], new V = Q_V [XV; 0] (panels, or full WY for wide sides
//               in the plain form)
//   finalize  : transpose V into the tile buffer, publish the new rank
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

#include "hcgb.h"

namespace hcgb {

constexpr int QR_NB = 16;          // Householder panel width (columns)
constexpr int MAX_JACOBI_SWEEPS = 40;

// FP64 tensor-core MMA (the only FP64 tensor path on sm_103a): {d0,d1} += a * b for an
// 8x8x4 tile.  Fragment layout (PTX ISA, mma.m8n8k4 .f64):
//   a : A[lane/4][lane%4]        (8 x 4, row)
//   b : B[lane%4][lane/4]        (4 x 8, col)
//   d : D[lane/4][2*(lane%4)+e]  (8 x 8), e = 0, 1
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// A set of NTH threads (whole warps) of one CTA that works on one update together: the thread's
// index in the team and the named barrier its members synchronise on (bar.sync id, NTH), so that
// two teams of one CTA never wait for each other.
template <int NTH>
struct Team {
    static constexpr int nth = NTH, ctas = 1;
    int tid, bar;
    __device__ __forceinline__ int warp() const { return tid >> 5; }
    __device__ __forceinline__ static constexpr int nw() { return NTH >> 5; }
    __device__ __forceinline__ static constexpr int warps_per_cta() { return NTH >> 5; }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NTH) : "memory"); }
};

// The NTH threads of each CTA of a thread-block cluster of CTAS as one team: threads are numbered through
// the cluster and sync() is the cluster's barrier, which also orders their global and distributed
// shared memory.  rank: this CTA's in the cluster.
template <int NTH, int CTAS>
struct ClusterTeam {
    static constexpr int nth = NTH * CTAS, ctas = CTAS, cta_threads = NTH;
    int tid, rank;
    __device__ __forceinline__ int warp() const { return tid >> 5; }
    __device__ __forceinline__ static constexpr int nw() { return (NTH * CTAS) >> 5; }
    __device__ __forceinline__ static constexpr int warps_per_cta() { return NTH >> 5; }
    __device__ __forceinline__ void sync() const {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ int cluster_rank() {
    int r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Address, in the generic space, of shared-memory object p of the cluster's CTA `rank`.
template <class T>
__device__ __forceinline__ T *cluster_map(T *p, int rank) {
    T *q;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
    return q;
}

// Every kernel launch of the library is counted (hcgb_kernel_launches reads the total).
void note_launch();

// Two launches on different updates run side by side in one stream: the first (the wide updates' clusters) lets the
// second start as soon as it runs itself; the second's first CTA ends only when the first is done, so what
// follows in the stream comes after both.  (A second stream would do, but the groups of a multiply already
// take every hardware queue: with one more stream a group the multiplies of few tiles took 30 % longer.)
__device__ __forceinline__ void let_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous_launch() {
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Launches the second of two such kernels (beside = whether there is a first one); cluster: its CTAs per cluster.
template <class... P, class... A>
void launch_beside(bool beside, int cluster, int grid, int block, size_t smem, cudaStream_t st, void (*kernel)(P...), A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    cfg.attrs = at;
    cfg.numAttrs = 0;
    if (beside) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = cluster;
        at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    cudaLaunchKernelEx(&cfg, kernel, args...);
    note_launch();
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// C = alpha * op(A) * op(B) + beta * C  (column-major; op 0 = N, 1 = T).  M <= 0: no job.
struct GemmJob {
    const double *A;
    const double *B;
    double *C;
    int M, N, K;
    int lda, ldb, ldc;
    int opA, opB;
    double alpha, beta;
    int oz;          // 1: computed on the 16-bit tensor cores by error-free splitting (oz_gemm.cu)
    int triA, triB;  // 1: the stored operand is read as unit lower trapezoidal (Householder vectors)
    int prec;        // 0: FP64-accurate (DMMA or oz); 1: TF32, 2: BF16 on tcgen05 (tc_gemm.cu)
};

constexpr int JOBS_PER_UPDATE = 6;  // job slots per update: 3 factor-product phases, 6 for the WY application

// Element (i, k) of op(A) with the job's op / unit-lower view (both GEMM kernels).
__device__ __forceinline__ double job_a(const GemmJob &jb, int i, int k) {
    const int r = jb.opA == 0 ? i : k, c = jb.opA == 0 ? k : i;
    if (jb.triA && r <= c) return r == c ? 1.0 : 0.0;
    return jb.A[r + (size_t) c * jb.lda];
}
__device__ __forceinline__ double job_b(const GemmJob &jb, int k, int j) {
    const int r = jb.opB == 0 ? k : j, c = jb.opB == 0 ? j : k;
    if (jb.triB && r <= c) return r == c ? 1.0 : 0.0;
    return jb.B[r + (size_t) c * jb.ldb];
}

// Precision of the factor products and of the WY Q-application products in arithmetic form `mode`.
__host__ __device__ inline int lowp_prec(int mode) { return mode == HCGB_TF32 ? 1 : (mode == HCGB_BF16 ? 2 : 0); }

// The job whose tile w is (sched: exclusive prefix sums of the jobs' tiles, njobs + 1 entries): a 32-way search by
// the whole warp, two or three dependent loads.
__device__ __forceinline__ int job_of_tile(const int *sched, int njobs, int w) {
    const int lane = threadIdx.x & 31;
    int lo = 0, n = njobs;  // sched[lo] <= w < sched[lo + n]
    while (n > 1) {
        const int step = (n + 31) >> 5, at = (lane + 1) * step;
        const unsigned below = __ballot_sync(0xffffffffu, at < n && sched[lo + at] <= w);
        const int skip = __popc(below) * step;
        lo += skip;
        n = n - skip < step ? n - skip : step;
    }
    return lo;
}

// Products worth the split: a 16 x 16 product takes both paths about as long (K = 512: 280 and 310 us for 608 of them;
// K = 64: 85 and 58), a 32 x 32 one is 2 and 1.2 times faster here.  Multiplies 11x11 nb=301, n=16384 and n=8192 at 1e-4:
// 68.5, 707 and 58.9 ms from 256 outputs and 24 reflectors on, 72.7, 719 and 61.0 from 2048 and 48 on.
constexpr int OZ_MIN_OUTPUTS = 256;
// The least for the products of an update with a dense C and for hcgb_dgemm: the split's error is relative to the
// row's and the column's maximum, an FP64 product's to the terms of each output.  Recompression truncates relative to
// the tile's norm; these results are the caller's as they are.
constexpr int OZ_MIN_OUTPUTS_DENSE = 2048;
__host__ __device__ inline bool oz_shape(int M, int N, int K, int min_outputs = OZ_MIN_OUTPUTS) {
    return K >= 16 && M >= 16 && N >= 8 && (long long) M * N >= min_outputs;
}

struct DevTile {
    double *data;  // U (rows x rank, ld rows), or the dense tile
    double *v;     // V region: data + rows * max_rank for a stored tile; the U buffer of the stored tile
                   // when this descriptor is the transpose of a compressed_vt tile (factors swapped)
    int *rank;
    int rows, cols, max_rank, kind;
};

struct DevUpdate {
    DevTile a, b, c;
    int uid;   // index of this update's record in the caller's hcgb_update_info array
    int dist;  // |i - j| of the C tile in a tile-matrix multiply (a feature of the rank predictor)
    int direct;  // 1: C = truncated SVD of the dense tile a (b unused, C at rank 0): the core alone
};

// Per-update bookkeeping written by the plan kernel and read by the later stages.
enum MetaField {
    META_STATUS = 0,
    META_CKIND,      // 1 when C is compressed (recompression needed)
    META_RA,
    META_RB,
    META_RC,
    META_SIDE,       // 0: stack [Cu | alpha Au], 1: stack [Cu | alpha Au (Av Bu)]
    META_K,          // columns of both stacks
    META_M,          // rows of C / of the U stack
    META_N,          // cols of C / rows of the V stack
    META_NEWRANK,
    META_SWEEPS,
    META_CORE_COLS,  // rows of R kept by the rank-revealing QR of the core
    META_KC_PRODUCT,  // core-kernel phase durations in units of 1024 SM cycles (diagnostics)
    META_KC_QRCP,
    META_KC_JACOBI,
    META_KC_FACTORS,
    META_WY,         // bit 0 / bit 1: the U / V factor's Q is applied in WY form (else apply_q_kernel)
    META_LSK,        // learned form: sketch width l (0: this update takes the plain recompression)
    META_SK_CK,      // learned form: CKIND, K and STATUS saved while the sketch / fallback passes run
    META_SK_K,
    META_SK_ST,
    META_SK_ACC,     // learned form: 1 when the sketch result passed the residual test
    META_INTS = 22
};

constexpr int WIDE_CTAS = 8;       // CTAs of a wide core's cluster
constexpr int WIDE_CLUSTERS = 19;  // clusters of a launch (152 SMs / 8)

// Device workspace: n slots of `slot_doubles` doubles plus an int meta block.
struct Workspace {
    double *base;
    int *meta;            // n * META_INTS
    int *order;           // optional (n ints): heavy-stage CTA b works on update order[b]
    size_t slot_doubles;
    int ld;               // leading dimension of every stack / temporary (>= rows, cols)
    int kmax;             // max columns of a stack
    int rmax;             // max rank of an A/B factor
    int conc = 1;         // launches like this one in flight at a time (the C-tile groups of a multiply)
    int k_wide, k_heavy;  // stack widths above which a core does not fit an SM's / half an SM's shared memory
    size_t off_ustack, off_vstack, off_tmp1, off_tmp2, off_tauu, off_tauv, off_tu, off_tv;
    size_t off_m, off_mcopy, off_xv, off_sigma, off_mixed;
    size_t mixed_floats;  // of the region at off_mixed: the preconditioner's columns of X and J, W
    size_t off_w;  // WY application: W_U, W_V (kmax x kmax each), present when built with wy
    size_t off_sk1, off_sk2, off_skaux;  // learned form: sketch stacks (ld x kmax each), residual estimate
    float *feat;   // learned form / feature sink: MLP_IN features per update (n x MLP_IN), or null
    float *pred;   // learned form: predicted log2(1 + rank) per update (n), or null

    __host__ __device__ double *slot(int s) const { return base + slot_doubles * (size_t) s; }
    // Update processed by CTA `b` of the QR / core / Q-application launches: largest first, so the
    // long updates of a launch start at once instead of after the short ones.
    __device__ int heavy(int b) const { return order ? order[b] : b; }
    // Key of an update in `order` (descending): its stack width when C is compressed.  The searches below hold only while
    // META_K and META_CKIND stand still: from launch_order to the end of that recompression.  The sketch passes of
    // the learned form rewrite both in between, and launch_order runs again before each of their recompressions.
    __device__ int key(int slot) const {
        const int *m = meta + (size_t) slot * META_INTS;
        return m[META_CKIND] ? m[META_K] : 0;
    }
    // Updates of `order` (of n) with a key above thr.
    __device__ int count_above(int n, int thr) const {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key(order[mid]) > thr) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    }
    // The first wide_updates(n) updates of `order` go to clusters of CTAs, stack QR and core: those whose core does not
    // fit an SM, and the heavy ones too while the launches in flight leave SMs for them.
    __device__ int wide_updates(int n) const {
        const int h = count_above(n, k_heavy);
        return (long) h * conc <= WIDE_CLUSTERS ? h : count_above(n, k_wide);
    }
};

// Layout of one workspace slot for stacks of up to `ld` rows and `kmax` columns; factor ranks
// up to `rmax`.  ddc_scratch reserves an ld x ld product for the DDC combination.  Host arithmetic alone (sizing needs no
// device); what launches on the workspace needs set_core_classes too.
Workspace make_workspace_layout(int ld, int kmax, int rmax, bool ddc_scratch, bool wy = false, bool learned = false);

struct Params {
    double accuracy;
    int truncated;
    int fixed_rank;
    int side_mode;   // 0: always the reference's [Cu | alpha Au]; 1: pick the smaller stack
    int mode;        // hcgb_mode: 0 plain FP64; 1 float-float QR / core / Q application; 2 / 3 TF32 / BF16
                     // factor products and Q-application products (QR, core, truncation in FP64)
    int oz;          // 1: large factor products on the 16-bit tensor cores (FP64-accurate splitting)
    int oz_min;      // outputs a product needs to go to the tensor cores (OZ_MIN_OUTPUTS by default)
    int wy_min;      // reflectors a side needs for the WY Q application (WY_MIN_REFLECTORS by default)
    int precond_min; // Jacobi columns a core needs for the FP32 preconditioning sweeps
    int sk_pct;      // learned form: sketch an update only when its sketch (with probes) is at most
                     // this percentage of its stack width
};

// Default of Params::sk_pct: a sketch of half the stack width halves the QR and Q-application work,
// which pays for the sketch products and its own QR; wider sketches cost more than they save.
constexpr int SKETCH_MAX_PCT = 50;

// Default of Params::precond_min: a 16-column core is about where the single-precision sweeps and the corrections
// cost what the FP64 sweeps do (25 columns: 348 kcycles against 930; 15 columns: 250 either way).
constexpr int PRECOND_MIN_COLS = 16;

// ---- launchers (stream-ordered, asynchronous) ----
void launch_plan(const DevUpdate *ups, int n, double alpha, double beta, Workspace ws, Params p, GemmJob *jobs,
                 cudaStream_t st);
void launch_stack(const DevUpdate *ups, int n, double alpha, double beta, Workspace ws, cudaStream_t st);
// ws.order <- updates sorted by decreasing stack width k (0 for a dense C; ties by index); needs
// ws.order != nullptr.  Run before every recompression (Workspace::key); the key ignores the status, which
// the core may change.
void launch_order(int n, Workspace ws, cudaStream_t st);
// out[i] = *ptrs[i] (device rank ints gathered for one host read).
void launch_gather_ranks(const int *const *ptrs, int n, int *out, cudaStream_t st);
// Batched products: sched = device scratch of 2 * njobs + 2 ints (tile prefix sums), njobs <= 4096.
// has_lowp: the list may hold TF32 / BF16 jobs (launches the tcgen05 kernel too).
void launch_gemm_jobs(const GemmJob *jobs, int njobs, int *sched, cudaStream_t st, bool has_lowp = false);
void launch_oz_gemm_jobs(const GemmJob *jobs, int njobs, const int *sched, int sms, cudaStream_t st);
void launch_tc_gemm_jobs(const GemmJob *jobs, int njobs, const int *sched, int sms, cudaStream_t st);
// Bounded mbarrier waits of the tcgen05 kernels that gave up (0 unless something else failed).
unsigned int tc_wait_timeouts();
unsigned int oz_wait_timeouts();
constexpr int MAX_JOBS_PER_LAUNCH = 4096;
constexpr int SCHED_INTS_PER_UPDATE = 16;  // >= (3 * 4n + 3) / n: one WY launch schedules 4n jobs, 3 tile lists
// Q application in full WY form (Q = I - V T V^T, T^-1 = striu(V^T V) + diag(1/tau)): jobs for
// the Grams, Y = V^T X and X -= V W, then the triangular solve T^-1 W = Y.  Used for the sides
// with at least WY_MIN_REFLECTORS reflectors (their products run on the tensor cores); the
// others keep the panel-wise apply_q_kernel, which skips the WY sides.  Plain form only: the mixed
// form's float-float panels are faster than either.
constexpr int WY_MIN_REFLECTORS = 24;
void launch_plan_wy(const DevUpdate *ups, int n, Workspace ws, Params p, GemmJob *jobs, cudaStream_t st);
void launch_wy_solve(int n, Workspace ws, cudaStream_t st);
void launch_qr(Workspace ws, int n, bool mixed, cudaStream_t st);
void launch_core_svd(const DevUpdate *ups, int n, Workspace ws, Params p, cudaStream_t st);
// Stack widths up to which a core fits a whole, half and a quarter of an SM's shared memory in launches of kmax (asks the
// device); set_core_classes fills the workspace's k_wide and k_heavy with the first two.
void core_classes(int kmax, int *whole, int *half, int *quarter);
void set_core_classes(Workspace *ws);
void launch_apply_q(const DevUpdate *ups, int n, Workspace ws, bool mixed, cudaStream_t st);
void launch_finalize(const DevUpdate *ups, int n, Workspace ws, hcgb_update_info *info, cudaStream_t st);
// FP64 throughput probes (TFLOP/s): tensor-core DMMA and SIMT DFMA.
int measure_fp64_peak(cudaStream_t st, double *dmma_tflops, double *dfma_tflops);
// DDC (dense A, dense B, compressed C): C <- full rank, U = alpha A B + beta Cu Cv, V = I.
void launch_ddc_finalize(const DevUpdate *ups, int n, Workspace ws, cudaStream_t st);
// dst (cols x rows, ld ldd) = src^T (src rows x cols, ld lds); one CTA.
void launch_transpose(const double *src, int lds, int rows, int cols, double *dst, int ldd, cudaStream_t st);

// Dense tile building blocks of a tile Cholesky (chol.cu).
void launch_trsm_panel(const double *L, int nb, int ldl, const DevTile *tiles, int count, int max_rank, cudaStream_t st);
void launch_fill_triangle(int uplo, int n, double *A, int lda, double value, cudaStream_t st);
// keep (n x n, or null): a copy of the triangle, from which launch_potrf_restore takes the columns from the failing
// one on (*info_dev = failed) back; without it they are left partly updated.
void launch_potrf(double *A, int n, int lda, int uplo, int *info_dev, double *keep, cudaStream_t st);
void launch_potrf_restore(double *A, int n, int lda, int uplo, int failed, const double *keep, cudaStream_t st);
void launch_trsm(int side, int uplo, int trans, int diag, int m, int n, double alpha, const double *A, int lda,
                 double *B, int ldb, cudaStream_t st);
void launch_syrk(int uplo, int trans, int n, int k, double alpha, const double *A, int lda, double beta, double *C,
                 int ldc, cudaStream_t st);

// Rank-trimmed packing of a tile list (pack.cu): offsets (n + 1) and the packed copy, or back.
void launch_pack(const DevTile *tiles, int n, long long *offsets, double *packed, bool unpack, cudaStream_t st);

// ---- learned form (learned.cu): features, sketch recompression and its fallback ----
// Per-update features (ws.feat, and sink[uid * MLP_IN ..] when sink != null); needs ws.feat.
void launch_features(const DevUpdate *ups, int n, Workspace ws, double accuracy, float *sink, cudaStream_t st);
// Sketch width per update from ws.pred (policy 0) or from the input ranks (policy 1), the jobs
// Z = V_s^T Omega (jobs[0 .. n)) and Y = U_s Z (jobs[n .. 2n)), and Omega itself.
void launch_sketch_plan(const DevUpdate *ups, int n, Workspace ws, Params p, int policy, unsigned long long seed,
                        GemmJob *jobs, cudaStream_t st);
// Householder QR of Y's first l columns, residual probe, explicit Q_Y; then the jobs W = U_s^T Q_Y
// (jobs[0 .. n)) and V' = V_s W (jobs[n .. 2n)).
void launch_sketch_qr(int n, Workspace ws, cudaStream_t st);
void launch_sketch_plan2(int n, Workspace ws, Params p, GemmJob *jobs, cudaStream_t st);
// stage 0: before the sketch pass; 1: residual test, before the fallback pass; 2: restore.
void launch_sketch_pass(int n, Workspace ws, Params p, int stage, cudaStream_t st);
void launch_learned_records(const DevUpdate *ups, int n, Workspace ws, hcgb_update_info *info, cudaStream_t st);

// ---- per-matrix operations of the HCoreKernels backend (backend.cu); asynchronous on st ----
void be_copy(cudaStream_t st, int trans, int m, int n, double alpha, const double *A, int lda, double *B, int ldb);
void be_lacpy(cudaStream_t st, int uplo, int m, int n, const double *A, int lda, double *B, int ldb);
void be_laset(cudaStream_t st, int uplo, int m, int n, double offdiag, double diag, double *A, int lda);
void be_scale_rows(cudaStream_t st, int rows, int cols, const double *s, double *A, int lda);
void be_symmetrize(cudaStream_t st, int uplo, int n, double *A, int lda);
void be_geqr2(cudaStream_t st, int m, int n, double *A, int lda, double *tau);
void be_org2r(cudaStream_t st, int m, int n, int k, double *A, int lda, const double *tau);
void be_orm2r(cudaStream_t st, int left, int trans, int m, int n, int k, const double *A, int lda, const double *tau,
              double *C, int ldc);
void be_trmm(cudaStream_t st, int left, int upper, int trans, int unit, int m, int n, double alpha, const double *A,
             int lda, const double *T, double *B, int ldb);
void be_jacobi_svd(cudaStream_t st, int rows, int cols, double *X, int ldx, double *V, int ldv, double tol, int *sweeps);
void be_svd_finish(cudaStream_t st, int rows, int cols, const double *X, int ldx, const double *V, int ldv, double *S,
                   double *U, int ldu, double *VT, int ldvt, int kk, int want_u, int want_vt, int transposed);

// ---- rank predictor of the learned form (mlp.cu) ----
constexpr int MLP_IN = 12, MLP_HIDDEN = 64;
constexpr int MLP_PARAMS = MLP_HIDDEN * MLP_IN + MLP_HIDDEN + MLP_HIDDEN * MLP_HIDDEN + MLP_HIDDEN + MLP_HIDDEN + 1;
struct RankModel {
    float *master = nullptr;  // FP32 master parameters, then grad, Adam m1, m2 (4 x MLP_PARAMS floats)
    float *grad = nullptr, *m1 = nullptr, *m2 = nullptr;
    __nv_bfloat16 *w = nullptr;  // BF16 weights read by the forward / backward kernels
    int adam_t = 0;
    int device = 0;
    int init(unsigned long long seed);
    int set_params(const float *host);
    int get_params(float *host) const;
    void release();
};
void launch_mlp_forward(const RankModel &m, const float *X, int n, float *Y, cudaStream_t st);
// grad += dL/dparams of L = inv_total * sum over samples (y - t)^2, *loss += sum (y - t)^2, for the
// samples idx[off .. off + n) (or rows off .. off + n when idx is null).
void launch_mlp_grad(const RankModel &m, const float *X, const float *T, const int *idx, int off, int n,
                     float inv_total, double *loss, cudaStream_t st);
void launch_adam(RankModel &m, float lr, cudaStream_t st);
void launch_targets_from_records(const hcgb_update_info *info, int n, float *T, int *keep, cudaStream_t st);

size_t qr_smem_bytes(int ld, int kmax);
size_t svd_smem_bytes(int kmax);

}  // namespace hcgb
