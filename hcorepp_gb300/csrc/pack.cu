// Rank-trimmed packing of a list of tiles: the device side of a TilePacker transfer
// (include/hcorepp/operators/interface/TilePacker.hpp:18-62 packs one tile at its full capacity,
// rows x max_rank + max_rank x cols; here a whole list is packed at once and a compressed tile
// contributes only the columns its rank uses).
//
// Packed format, tiles in list order, each starting at offsets[t] (doubles):
//   dense:           rows x cols, column-major
//   compressed:      U (rows x rank, ld rows) followed by V (rank x cols, ld rank)
//   compressed_vt:   U (rows x rank, ld rows) followed by W = V^T (cols x rank, ld cols)
// In the tile buffers both factor blocks are contiguous (U's leading dimension is rows, the V
// region's is rank for compressed and cols for compressed_vt), so every tile is at most two
// contiguous copies.  offsets[count] is the total.
#include "internal.cuh"

namespace hcgb {

namespace {

__device__ __forceinline__ long long packed_doubles(const DevTile &t) {
    if (!t.kind) return (long long) t.rows * t.cols;
    const long long r = *t.rank;
    return r * (t.rows + t.cols);
}

constexpr int PACK_CTAS = 3648;

// offsets[0..n] = exclusive prefix sum of the packed sizes; one CTA: every thread sums a
// contiguous run of tiles, a Hillis-Steele scan combines the runs.
__global__ void __launch_bounds__(1024) pack_offsets_kernel(const DevTile *tiles, int n, long long *offsets) {
    __shared__ long long part[1024];
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int b0 = threadIdx.x * per;
    const int b1 = b0 + per < n ? b0 + per : n;
    long long s = 0;
    for (int i = b0; i < b1; i++) s += packed_doubles(tiles[i]);
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < (int) blockDim.x; o <<= 1) {
        const long long v = (int) threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    long long run = threadIdx.x ? part[threadIdx.x - 1] : 0;
    for (int i = b0; i < b1; i++) {
        offsets[i] = run;
        run += packed_doubles(tiles[i]);
    }
    if (threadIdx.x == blockDim.x - 1) offsets[n] = part[blockDim.x - 1];
}

// The part-th of `parts` shares of a copy, eight values a thread in flight.
__device__ __forceinline__ void copy_run(const double *__restrict__ src, double *__restrict__ dst, long long len,
                                         int part, int parts) {
    constexpr int U = 8;
    const long long step = (long long) blockDim.x * U, share = (len + parts - 1) / parts;
    const long long end = share * (part + 1) < len ? share * (part + 1) : len;
    for (long long e0 = share * part; e0 < end; e0 += step) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long e = e0 + threadIdx.x + (long long) u * blockDim.x;
            if (e < end) v[u] = src[e];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long e = e0 + threadIdx.x + (long long) u * blockDim.x;
            if (e < end) dst[e] = v[u];
        }
    }
}

// gridDim.y CTAs per tile, a share of its values each: unpack = 0 copies the tile's used part into the packed
// buffer, 1 back.  Bound by memory; with one CTA a tile the 2 MB of a dense 512 x 512 tile set the time
// (a 16 x 16-tile matrix out and back in: 950 us).
__global__ void __launch_bounds__(256) pack_kernel(const DevTile *tiles, int n, const long long *offsets,
                                                   double *packed, int unpack) {
    const int t = blockIdx.x;
    if (t >= n) return;
    const DevTile d = tiles[t];
    double *p = packed + offsets[t];
    const long long r = d.kind ? *d.rank : 0;
    const long long lu = d.kind ? r * d.rows : (long long) d.rows * d.cols, lv = r * d.cols;
    if (unpack) {
        copy_run(p, d.data, lu, blockIdx.y, gridDim.y);
        if (lv > 0) copy_run(p + lu, d.v, lv, blockIdx.y, gridDim.y);
    } else {
        copy_run(d.data, p, lu, blockIdx.y, gridDim.y);
        if (lv > 0) copy_run(d.v, p + lu, lv, blockIdx.y, gridDim.y);
    }
}

}  // namespace

void launch_pack(const DevTile *tiles, int n, long long *offsets, double *packed, bool unpack, cudaStream_t st) {
    { pack_offsets_kernel<<<1, 1024, 0, st>>>(tiles, n, offsets); note_launch(); }
    // enough CTAs for the whole GPU whatever the number of tiles (PACK_CTAS: 152 SMs x 8 CTAs, three times over)
    const int split = PACK_CTAS / n < 1 ? 1 : (PACK_CTAS / n < 128 ? PACK_CTAS / n : 128);
    { pack_kernel<<<dim3(n, split), 256, 0, st>>>(tiles, n, offsets, packed, unpack ? 1 : 0); note_launch(); }
}

}  // namespace hcgb
