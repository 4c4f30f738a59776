// FP64 factor products on the fifth-generation tensor cores by error-free splitting (the Ozaki
// scheme), with tcgen05.mma (kind::f16, FP32 accumulation in tensor memory).
//
// The GB300's FP64 pipe (SIMT or DMMA) delivers ~1.1 TFLOP/s, its FP16 tensor cores ~2 PFLOP/s.
// A product C = op(A) op(B) is computed exactly enough for FP64 work as follows:
//   * every row i of op(A) gets the exponent e_i with max_k |A_ik| < 2^e_i, every column j of
//     op(B) the exponent f_j with max_k |B_kj| < 2^f_j;
//   * each element becomes a 56-bit fixed-point integer relative to its group's exponent (rounded
//     to nearest; the rounding error is 2^-57 of the group maximum) and is cut into S = 8 balanced
//     base-128 digits, A = sum_s 2^(e_i - 7 (s + 1)) A^(s), |A^(s)| <= 64 for s > 0 and <= 128 for
//     s = 0, all exact in FP16;
//   * the plane products A^(s) B^(t) are integers; the pairs of one level L = s + t (at most 8
//     per k, each below 2^13 but the (0, 0) one) sum to less than 2^15 per k, so over 128 k the
//     FP32 accumulators of a level hold them exactly (< 2^22) and an FP32 add of 1.5 * 2^23 exposes
//     them as integers in the low mantissa bits;
//   * levels L = s + t <= S - 1 are kept (36 plane pairs; the dropped ones are below 2^-56 of
//     max|A_i| max|B_j| per k, under FP64's own worst-case bound); every 128 k the eight level
//     accumulators are read out of tensor memory and added into two 64-bit integers (levels 0-3 and
//     4-7, each shifted to a common scale), which stay exact for k up to 2^16, and the tile ends with
//     C_ij = 2^(e_i + f_j) (hi 2^-35 + lo 2^-63);
//   * outputs of a row or column that holds a NaN or an infinity are FP64 products.
// Tensor memory holds the eight level accumulators of a 128 x 64 output tile (512 columns).  The sixteen warps cut
// 32-wide K chunks into digit planes, two shared-memory stages in turn, and read the accumulators out; a thread of the
// last one issues the 72 MMAs (36 pairs x 2 k-steps of 16) of a chunk when it is filled.  They meet on mbarriers
// only (every wait bounded).
//
// What bounds it is the splitting, not the tensor cores: every operand element becomes eight FP16 digits.  A
// bias of 64 in every digit makes the balanced digits independent bit fields (no carry from digit to digit),
// two of them at a time become halves by one exact subtraction (1024 + d as a bit pattern), a thread takes
// eight consecutive K of a row, so a plane costs one 16-byte store without bank conflicts, and rows beyond
// the job are left alone (they only reach accumulators nobody reads).  Sixteen warps, four to a
// sub-partition, hide the latencies; sums and outputs are put together by integer operations, one FP64
// instruction an output for beta C.  Sixteen warps instead of eight and this
// splitting took the products of a 32 x 32-tile multiply (nb = 512) from 108 to 86 ms and its Q application
// from 214 to 184.
#include <cuda_fp16.h>

#include <type_traits>

#include "internal.cuh"
#include "tcgen05.cuh"

namespace hcgb {

namespace {

constexpr int OZ_S = 8;                 // digit planes per operand
constexpr int OZ_B = 7;                 // bits per digit
constexpr int OZ_W = OZ_S * OZ_B;       // fixed-point width (56 bits)
static_assert(OZ_W >= 53, "the digit planes must cover a double's 53-bit significand");
constexpr int OZ_TM = 128, OZ_TN = 64;  // output tile per CTA (UMMA M = 128, N = 64)
constexpr int OZ_KC = 32;               // K elements per shared-memory stage (64 bytes per row and plane)
constexpr int OZ_KB = OZ_KC * 2 / 16;   // core matrices along K per stage (4)
constexpr int OZ_FLUSH = 4;             // stages per exact read-out of the level accumulators (128 k)
constexpr int OZ_THREADS = 512;         // 16 warps
constexpr int OZ_A_PLANE = OZ_TM * OZ_KC * 2;   // 8 KB
constexpr int OZ_B_PLANE = OZ_TN * OZ_KC * 2;   // 4 KB
constexpr int OZ_STAGE = OZ_S * (OZ_A_PLANE + OZ_B_PLANE);  // 96 KB
static_assert(OZ_TM * OZ_TN * 8 <= 2 * OZ_STAGE, "a tile's outputs fit the stages");
constexpr int OZ_SMEM = 2 * OZ_STAGE + 1024;
constexpr int OZ_TMEM_COLS = OZ_S * OZ_TN;  // 512: one 64-column accumulator per level
constexpr int OZ_NOGROUP = -1100;       // exponent of an all-zero group
constexpr int OZ_NONFINITE = 1 << 20;   // exponent of a group with a NaN or an infinity (cut to zeros)

__device__ unsigned int g_oz_wait_timeouts = 0;

// Biased exponent field of |x| (0 for zero and subnormals).
__device__ __forceinline__ int exp_field(double x) {
    return (int) ((__double_as_longlong(x) >> 52) & 0x7ff);
}

// The 56-bit fixed-point integer of x relative to the group exponent e (|x| < 2^e), v = round(x 2^(56 - e)), plus
// 64 in each digit but the leading one and 128 in that: digit s is the 7-bit field at 7 (7 - s) minus 64, the
// leading digit what lies above bit 49 minus 128: d[1..7] in [-64, 63], d[0] in [-128, 128].  Subnormals
// count as zero.
constexpr unsigned long long OZ_BIAS = (128ull << 49) | (64ull << 42) | (64ull << 35) | (64ull << 28) | (64ull << 21) |
                                       (64ull << 14) | (64ull << 7) | 64ull;
__device__ __forceinline__ unsigned long long oz_biased(double x, int e) {
    const long long bits = __double_as_longlong(x);
    const int E = (int) ((bits >> 52) & 0x7ff);
    long long u = 0;
    if (E != 0 && e > OZ_NOGROUP) {
        const long long M = (bits & 0xfffffffffffffLL) | (1LL << 52);
        const int sh = E - 1019 - e;  // x * 2^(56 - e) = M * 2^sh, sh <= 3
        if (sh >= 0) u = M << sh;
        else if (sh > -64) u = (M + (1LL << (-sh - 1))) >> (-sh);
    }
    return (unsigned long long) (bits < 0 ? -u : u) + OZ_BIAS;
}

// Digits `s` of two biased integers as a pair of halves.
template <int S>
__device__ __forceinline__ uint32_t oz_digit_pair(unsigned long long u0, unsigned long long u1) {
    constexpr int SHIFT = OZ_B * (OZ_S - 1 - S);
    constexpr uint32_t MASK = S ? 127u : 511u;
    const uint32_t x0 = (uint32_t) (u0 >> SHIFT) & MASK, x1 = (uint32_t) (u1 >> SHIFT) & MASK;
    const uint32_t m = x0 | (x1 << 16) | 0x64006400u;  // 1024 + x as FP16
    const uint32_t off = S ? 0x64406440u : 0x64806480u;  // 1024 + 64, 1024 + 128
    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&m), *reinterpret_cast<const __half2 *>(&off));
    return *reinterpret_cast<const uint32_t *>(&d);
}

// Byte offset of (row r, K element kk of the stage) inside one plane (core-matrix layout, 2-byte
// elements, OZ_KB core matrices along K).
__device__ __forceinline__ int oz_off(int r, int kk) {
    return ((r >> 3) * OZ_KB + (kk >> 3)) * 128 + (r & 7) * 16 + (kk & 7) * 2;
}

// (hi 2^28 + lo) 2^(e - 63) as a double, rounded once (to nearest even), by integer operations without branches
// (a normal result; the rare others through ldexp).
__device__ __forceinline__ double oz_value(long long hi, long long lo, int e) {
    long long t = hi + (lo >> 28);
    uint32_t r = (uint32_t) lo & 0xfffffffu;  // the number is t 2^28 + r
    const bool neg = t < 0;
    t = neg ? ~t + (r == 0 ? 1 : 0) : t;
    r = neg ? (0u - r) & 0xfffffffu : r;
    // |number| 2^4 as three words, the leading bit shifted to the top
    uint32_t w2 = (uint32_t) ((unsigned long long) t >> 32), w1 = (uint32_t) t, w0 = r << 4;
    int n = 0;
    const bool z2 = w2 == 0;
    w2 = z2 ? w1 : w2;
    w1 = z2 ? w0 : w1;
    w0 = z2 ? 0u : w0;
    n += z2 ? 32 : 0;
    const bool z1 = w2 == 0;
    w2 = z1 ? w1 : w2;
    w1 = z1 ? w0 : w1;
    w0 = z1 ? 0u : w0;
    n += z1 ? 32 : 0;
    const int c = __clz(w2) & 31;
    const bool zero = w2 == 0;
    w2 = __funnelshift_l(w1, w2, c);
    w1 = __funnelshift_l(w0, w1, c);
    w0 <<= c;
    n += c;
    // the leading bit stands for 2^(91 - n) of the number
    const uint32_t rest = w1 & 0x7ffu;
    unsigned long long m = ((unsigned long long) w2 << 21) | (w1 >> 11);
    m += (rest > 0x400u || (rest == 0x400u && (w0 != 0 || (m & 1)))) ? 1 : 0;
    const int field = 91 - n + e - 63 + 1023;
    const unsigned long long bits = ((unsigned long long) (field - 1) << 52) + m;
    double v = zero ? 0.0 : __longlong_as_double((long long) bits);
    if (!zero && (field <= 0 || field >= 2046)) v = ldexp((double) m, field - 1023 - 52);
    return neg ? -v : v;
}

// Elements k0 .. k0 + NK - 1 of row g of op(A) (IS_A) or of column g of op(B), zero beyond K.
template <bool IS_A, int NK>
__device__ __forceinline__ void load_run(const GemmJob &jb, int g, int k0, double (&v)[NK]) {
    const int op = IS_A ? jb.opA : jb.opB, ld = IS_A ? jb.lda : jb.ldb, tri = IS_A ? jb.triA : jb.triB;
    const bool kcol = IS_A ? op == 0 : op != 0;  // k is the stored column index
    const double *p = (IS_A ? jb.A : jb.B) + (kcol ? (size_t) g + (size_t) k0 * ld : (size_t) k0 + (size_t) g * ld);
    const size_t step = kcol ? (size_t) ld : 1;
#pragma unroll
    for (int q = 0; q < NK; q++) {
        v[q] = k0 + q < jb.K ? p[step * q] : 0.0;
        if (tri) {
            const int r = kcol ? g : k0 + q, c = kcol ? k0 + q : g;
            if (r <= c && k0 + q < jb.K) v[q] = r == c ? 1.0 : 0.0;
        }
    }
}

// NK (4 or 8) consecutive K elements of row r of the tile (row g of the operand) into the eight digit planes.
template <int NK>
__device__ __forceinline__ void split_run(const double (&v)[NK], int e, unsigned char *at, int plane_bytes) {
    unsigned long long u[NK];
#pragma unroll
    for (int q = 0; q < NK; q++) u[q] = oz_biased(v[q], e);
    auto plane = [&](auto tag) {
        constexpr int S = decltype(tag)::value;
        uint32_t w[NK / 2];
#pragma unroll
        for (int q = 0; q < NK / 2; q++) w[q] = oz_digit_pair<S>(u[2 * q], u[2 * q + 1]);
        unsigned char *d = at + S * plane_bytes;
        if constexpr (NK == 8) *reinterpret_cast<uint4 *>(d) = make_uint4(w[0], w[1], w[2], w[3]);
        else *reinterpret_cast<uint2 *>(d) = make_uint2(w[0], w[1]);
    };
    plane(std::integral_constant<int, 0>{});
    plane(std::integral_constant<int, 1>{});
    plane(std::integral_constant<int, 2>{});
    plane(std::integral_constant<int, 3>{});
    plane(std::integral_constant<int, 4>{});
    plane(std::integral_constant<int, 5>{});
    plane(std::integral_constant<int, 6>{});
    plane(std::integral_constant<int, 7>{});
}

// Barriers of the CTA: full[2] (the sixteen warps have filled a stage), empty[2] (the MMAs have read it: a commit),
// read (the sixteen warps have read the accumulators).
struct OzBarriers {
    uint32_t full, empty, read;
};

// One 128 x 64 output tile of one job.  chunks / windows: 32-wide K chunks and read-out windows of the CTA's earlier
// tiles; chunk t fills stage t & 1 for the (t >> 1)-th time.
__device__ void oz_tile(const GemmJob &jb, int tile, unsigned char *stage0, uint32_t tmem, const OzBarriers &bars,
                        int &chunks, int &windows, int *ea, int *eb, int *special) {
    const int ntm = (jb.M + OZ_TM - 1) / OZ_TM;
    const int m0 = (tile % ntm) * OZ_TM, n0 = (tile / ntm) * OZ_TN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows = jb.M - m0 < OZ_TM ? jb.M - m0 : OZ_TM, cols = jb.N - n0 < OZ_TN ? jb.N - n0 : OZ_TN;
    const uint32_t idesc = tc::instr_desc(tc::FMT_F16, OZ_TM, (cols + 15) & ~15);

    // 1. Group exponents over all of K, largest exponent field per row of op(A) and column of op(B); the
    //    threads of a group are laid out so that consecutive lanes read consecutive addresses.
    if (tid == 0) *special = 0;
    if (tid < OZ_TM) ea[tid] = 0;
    else if (tid < OZ_TM + OZ_TN) eb[tid - OZ_TM] = 0;
    __syncthreads();
    auto exponents = [&](auto is_a, int count, int *out) {
        constexpr bool IS_A = decltype(is_a)::value;
        const bool kfast = IS_A ? jb.opA != 0 : jb.opB == 0;
        int groups = 16;  // few rows: more threads each
        while (groups < count) groups <<= 1;
        const int per = OZ_THREADS / groups;
        const int g = kfast ? tid / per : tid % groups, part = kfast ? tid % per : tid / groups;
        if (g >= count) return;
        int top = 0;
#pragma unroll 4
        for (int k = 4 * part; k < jb.K; k += 4 * per) {
            double v[4];
            load_run<IS_A, 4>(jb, (IS_A ? m0 : n0) + g, k, v);
#pragma unroll
            for (int q = 0; q < 4; q++) top = max(top, exp_field(v[q]));
        }
        if (top) atomicMax(out + g, top);
    };
    exponents(std::true_type{}, rows, ea);
    exponents(std::false_type{}, cols, eb);
    __syncthreads();
    if (tid < OZ_TM + OZ_TN) {
        int *e = tid < OZ_TM ? ea + tid : eb + (tid - OZ_TM);
        const int top = *e;
        *e = top == 0x7ff ? OZ_NONFINITE : (top ? top - 1022 : OZ_NOGROUP);
        if (top == 0x7ff) *special = 1;
    }
    __syncthreads();

    // This thread's share of the read-out: TMEM lanes 32 (warp % 4) .. (rows), columns 16 (warp / 4) ..
    const int q = warp & 3, h = warp >> 2;
    const bool reads = q * 32 < rows && h * 16 < cols;
    unsigned long long hi[16], lo[16];  // levels 0-3 at scale 2^-35, levels 4-7 at scale 2^-63
#pragma unroll
    for (int j = 0; j < 16; j++) hi[j] = lo[j] = 0;
    bool ok = true;
    // A level sum iv appears as the bit pattern 0x4B400000 + iv of iv + 1.5 2^23; the pattern is added with the
    // level's weight, what the constant contributes is taken off at the end.
    auto readout = [&]() {
        if (reads) {
#pragma unroll 1
            for (int l = 0; l < OZ_S; l++) {
                float v[16];
                tc::tmem_ld16(tmem + ((uint32_t) (q * 32) << 16) + (uint32_t) (l * OZ_TN + h * 16), v);
                const uint32_t weight = 1u << (OZ_B * ((l < 4 ? 3 : 7) - l));
                if (l < 4) {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        hi[j] += (unsigned long long) __float_as_uint(v[j] + 12582912.0f) * weight;
                } else {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        lo[j] += (unsigned long long) __float_as_uint(v[j] + 12582912.0f) * weight;
                }
            }
        }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bars.read);  // the next window's MMAs may overwrite the accumulators
    };

    // this thread's runs: eight K of a row of A, four of a column of B (see oz_off for the layout)
    const bool ka = jb.opA != 0;
    const int ra = ka ? tid >> 2 : tid & 127, ca = ka ? tid & 3 : tid >> 7;
    const int rb = (tid & 7) + 8 * (tid >> 6), cb = ((tid >> 4) & 3) * 8 + ((tid >> 3) & 1) * 4;
    const int nchunks = (jb.K + OZ_KC - 1) / OZ_KC, nwindows = (nchunks + OZ_FLUSH - 1) / OZ_FLUSH;
    // the MMAs of chunk c, by one thread
    auto issue = [&](int c) {
        const int t = chunks + c, buf = t & 1, fill = t >> 1, window = windows + c / OZ_FLUSH;
        const bool first = (c % OZ_FLUSH) == 0;  // accumulators restart after every read-out
        ok &= tc::mbar_wait(bars.full + 8 * buf, fill & 1);
        if (first && window > 0) ok &= tc::mbar_wait(bars.read, (window - 1) & 1);
        tc::fence_after();
        unsigned char *sa = stage0 + buf * OZ_STAGE, *sb = sa + OZ_S * OZ_A_PLANE;
        const uint64_t ad = tc::smem_desc(tc::smem_u32(sa), 128, OZ_KB * 128);
        const uint64_t bd = tc::smem_desc(tc::smem_u32(sb), 128, OZ_KB * 128);
#pragma unroll
        for (int ks = 0; ks < OZ_KC / 16; ks++)
#pragma unroll
            for (int s = 0; s < OZ_S; s++)
#pragma unroll
                for (int u = 0; u < OZ_S - s; u++) {
                    // The first MMA into level L of a read-out window overwrites it: in this order
                    // that is the pair (0, L) of the window's first k-step.
                    const bool overwrite = first && ks == 0 && s == 0;
                    tc::mma_f16(tmem + (uint32_t) ((s + u) * OZ_TN), ad + ((s * OZ_A_PLANE + ks * 256) >> 4),
                                bd + ((u * OZ_B_PLANE + ks * 256) >> 4), idesc, overwrite ? 0u : 1u);
                }
        tc::commit(bars.empty + 8 * buf);
    };
    double va[8], vb[4];  // the next chunk's runs, loaded while this one's products are issued and read out
    auto load = [&](int c) {
        if (ra < rows) load_run<true, 8>(jb, m0 + ra, c * OZ_KC + 8 * ca, va);
        if (rb < cols) load_run<false, 4>(jb, n0 + rb, c * OZ_KC + cb, vb);
    };
    if (nchunks > 0) load(0);
    for (int c = 0; c < nchunks; c++) {
        const int t = chunks + c, buf = t & 1, fill = t >> 1;
        unsigned char *sa = stage0 + buf * OZ_STAGE, *sb = sa + OZ_S * OZ_A_PLANE;
        if (fill > 0) ok &= tc::mbar_wait(bars.empty + 8 * buf, (fill - 1) & 1);
        if (ra < rows) split_run<8>(va, ea[ra], sa + oz_off(ra, 8 * ca), OZ_A_PLANE);
        if (rb < cols) split_run<4>(vb, eb[rb], sb + oz_off(rb, cb), OZ_B_PLANE);
        tc::fence_smem_to_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bars.full + 8 * buf);
        if (c + 1 < nchunks) load(c + 1);
        if (__shfl_sync(0xffffffffu, warp, 0) == OZ_THREADS / 32 - 1) {  // uniform, as the MMAs' operands must be
            if (tc::elect_one()) issue(c);
            __syncwarp();
        }
        if ((c + 1) % OZ_FLUSH == 0 || c + 1 == nchunks) {
            ok &= tc::mbar_wait(bars.empty + 8 * buf, fill & 1);  // this commit covers every earlier MMA
            tc::fence_after();
            readout();
        }
    }
    chunks += nchunks;
    windows += nwindows;
    if (!__all_sync(0xffffffffu, ok) && lane == 0) atomicAdd(&g_oz_wait_timeouts, 1u);  // the MMAs' waits are one lane's

    // Outputs of a row or column with a NaN or an infinity, as an FP64 product gives them: put aside in the stages, which the
    // MMAs have read, and stored over what the epilogue makes of them.  (A test an output in the epilogue cost the
    // products 2 %.)
    double *stash = reinterpret_cast<double *>(stage0);
    if (*special) {
        for (int e = tid; e < rows * cols; e += OZ_THREADS) {
            const int r = e % rows, c = e / rows;
            if (ea[r] + eb[c] < OZ_NONFINITE / 2) continue;
            double v = 0.0;
            for (int k = 0; k < jb.K; k++) v = fma(job_a(jb, m0 + r, k), job_b(jb, k, n0 + c), v);
            v *= jb.alpha;
            if (jb.beta != 0.0) v = fma(jb.beta, jb.C[m0 + r + (size_t) (n0 + c) * jb.ldc], v);
            stash[e] = v;
        }
        __syncthreads();
    }

    // Epilogue: C = alpha * product + beta * C, one row per thread, 16 columns.
    const int row_l = q * 32 + lane;
    if (reads && row_l < rows) {
        const unsigned long long constant =
            (unsigned long long) nwindows * 0x4B400000ull * ((1ull << 21) + (1ull << 14) + (1ull << 7) + 1ull);
        const bool scale = jb.alpha != 1.0 && jb.alpha != -1.0, negate = jb.alpha == -1.0, accum = jb.beta != 0.0;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int cl = h * 16 + j;
            if (cl < cols) {
                double *cp = jb.C + m0 + row_l + (size_t) (n0 + cl) * jb.ldc;
                double v = 0.0;
                if (jb.K > 0) v = oz_value((long long) (hi[j] - constant), (long long) (lo[j] - constant), ea[row_l] + eb[cl]);
                if (negate) v = -v;
                if (scale) v *= jb.alpha;
                if (accum) v = fma(jb.beta, *cp, v);
                *cp = v;
            }
        }
    }
    if (*special) {
        __syncthreads();
        for (int e = tid; e < rows * cols; e += OZ_THREADS)
            if (ea[e % rows] + eb[e / rows] >= OZ_NONFINITE / 2)
                jb.C[m0 + e % rows + (size_t) (n0 + e / rows) * jb.ldc] = stash[e];
    }
    __syncthreads();  // ea / eb are rewritten by the next tile
}

// Tiles of the jobs marked oz, compacted (sched: exclusive prefix of tiles per job, njobs + 1
// entries); a grid sized to the GPU strides over them.
__global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm_jobs_kernel(const GemmJob *jobs, int njobs, const int *sched) {
    extern __shared__ __align__(1024) unsigned char oz_smem_raw[];
    __shared__ __align__(8) unsigned long long mbar[5];
    __shared__ uint32_t tmem_slot;
    __shared__ int ea[OZ_TM], eb[OZ_TN], special;
    unsigned char *stage0 = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(oz_smem_raw) + 1023) & ~uintptr_t(1023));
    const int total = sched[njobs];
    if (blockIdx.x >= total) return;  // whole CTA leaves before any TMEM or barrier is set up
    const uint32_t mbar0 = tc::smem_u32(&mbar[0]);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(mbar0 + 8 * b, OZ_THREADS / 32);
            tc::mbar_init(mbar0 + 16 + 8 * b, 1);
        }
        tc::mbar_init(mbar0 + 32, OZ_THREADS / 32);
    }
    if ((threadIdx.x >> 5) == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), OZ_TMEM_COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const OzBarriers bars{mbar0, mbar0 + 16, mbar0 + 32};
    int chunks = 0, windows = 0;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int lo = job_of_tile(sched, njobs, w);
        const GemmJob jb = jobs[lo];
        oz_tile(jb, w - sched[lo], stage0, tmem, bars, chunks, windows, ea, eb, &special);
    }
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) tc::tmem_free(tmem, OZ_TMEM_COLS);
}

}  // namespace

void launch_oz_gemm_jobs(const GemmJob *jobs, int njobs, const int *sched, int sms, cudaStream_t st) {
    if (njobs <= 0) return;
    cudaFuncSetAttribute(oz_gemm_jobs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM);
    { oz_gemm_jobs_kernel<<<sms, OZ_THREADS, OZ_SMEM, st>>>(jobs, njobs, sched); note_launch(); }
}

unsigned int oz_wait_timeouts() {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_oz_wait_timeouts, sizeof(v));
    return v;
}

}  // namespace hcgb
