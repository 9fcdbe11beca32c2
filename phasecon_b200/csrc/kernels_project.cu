// Layout conversions and the sparse forward / back projectors.
//
// Forward projection (replaces initErrorSinogam, MBIR_4D/XT_ICD_update.c:651-712,
// and forward_project_voxel_AMat1D, XT_ForwardProject.c:44-61): column-driven,
// FP64 accumulation in an L2-resident FP64 image of the sinogram, rounded to
// float once: e = y - A x (or A x when no y is given). The A value is used
// unscaled, as the reference does here (the voxel update scales it by
// delta_t, XT_VoxUpdate.c:61).
//
// Back projection (the adjoint, A^T s): lanes over detector rows and neighbouring
// columns, FP64 accumulation over the frame's views (of FP32 sums over groups of
// four views where the records are one 16-byte word), then a sum over the
// z_overlap rows of each voxel slice.
#include <algorithm>

#include "mbir_internal.h"

namespace mbirgpu {

// [N_p][N_t][N_r] (the ABI's [view][row][col]) -> [N_p][N_r][N_t]
__global__ void transpose_rows_cols(const float *__restrict__ in, float *__restrict__ out, int N_t, int N_r)
{
    __shared__ float tile[32][33];
    const size_t base = (size_t)blockIdx.z * N_t * N_r;
    const int r0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int t = t0 + i, r = r0 + threadIdx.x;
        if (t < N_t && r < N_r) tile[i][threadIdx.x] = in[base + (size_t)t * N_r + r];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int r = r0 + i, t = t0 + threadIdx.x;
        if (t < N_t && r < N_r) out[base + (size_t)r * N_t + t] = tile[threadIdx.x][i];
    }
}

void launch_transpose_sino(const float *in, float *out, int N_p, int N_t, int N_r, cudaStream_t st)
{
    dim3 grid((N_r + 31) / 32, (N_t + 31) / 32, N_p), block(32, 8);
    transpose_rows_cols<<<grid, block, 0, st>>>(in, out, N_t, N_r);
}

void launch_untranspose_sino(const float *in, float *out, int N_p, int N_r, int N_t, cudaStream_t st)
{
    // [N_p][N_r][N_t] -> [N_p][N_t][N_r] is the same transpose with the roles swapped
    dim3 grid((N_t + 31) / 32, (N_r + 31) / 32, N_p), block(32, 8);
    transpose_rows_cols<<<grid, block, 0, st>>>(in, out, N_r, N_t);
}

// [T][Z][Y*X] <-> [T][Y*X][Z]
void launch_vol_to_zfast(const float *in, float *out, int N_time, int N_z, int N_y, int N_x, cudaStream_t st)
{
    const int nxy = N_y * N_x;
    dim3 grid((nxy + 31) / 32, (N_z + 31) / 32, N_time), block(32, 8);
    transpose_rows_cols<<<grid, block, 0, st>>>(in, out, N_z, nxy);
}

void launch_zfast_to_vol(const float *in, float *out, int N_time, int N_z, int N_y, int N_x, cudaStream_t st)
{
    const int nxy = N_y * N_x;
    dim3 grid((N_z + 31) / 32, (nxy + 31) / 32, N_time), block(32, 8);
    transpose_rows_cols<<<grid, block, 0, st>>>(in, out, nxy, N_z);
}

// Forward projection of a tile: a CTA owns a tile of voxel columns of one frame
// (and one 32-row chunk; lane = detector row), its warps take the frame's views in
// pairs. For one view a tile's A entries fall on a narrow band of detector channels,
// and the warp goes through the band channel by channel: the columns whose first
// entry is on channel o (a ballot finds them) add their products to the W FP64
// registers of channels o .. o + W - 1, then channel o is complete, goes to the FP64
// sinogram image as one reduction of a warp, and the registers move up. A column's
// weights are converted once, by the lane that loads its record, and read back from
// shared memory by all lanes, as are the voxels.
//
// What bounds it: shared-memory wavefronts (4 a record: its voxels, its weights) and
// issue (23 instructions a record), 72 % and 64 % busy; 16 B of table a record come
// from HBM. 256 x 256 x 32 x 8 voxels, 1024 views: 2.13 ms (the
// table's 1.07 GB alone would take 0.16); with the band in shared memory instead of registers (4
// wavefronts more for each entry) and tiles of 32 columns (twice the reductions)
// 4.27. Two CTAs an SM instead of three 2.37, two columns at a time 2.28. Columns
// whose voxels are all zero are skipped.
constexpr int kFpWarps = 8;

// KW: 16-byte words per A record (1, 2, 3 for voxel scale 1, 2, 4): up to 4 KW - 1
// entries. The tile shrinks with KW: its weights take the same shared memory.
template <int KW>
struct FpTile {
    static constexpr int W = 4 * KW - 1;
    static constexpr int G = KW == 1 ? 4 : KW == 2 ? 2 : 1;  // groups of 32 columns
    static constexpr int TX = KW == 1 ? 16 : 8, TY = KW == 3 ? 4 : 8;
    static constexpr int cols = 32 * G;
    static_assert(TX * TY == cols, "a lane per column of a group");
    static constexpr size_t bytes = sizeof(double) * cols * (32 + kFpWarps * (W + 1));
};

template <int KW>
__global__ void __launch_bounds__(kFpWarps * 32, 3) forward_project_kernel(Geom g, const uint32_t *__restrict__ table,
                                                                          const int32_t *__restrict__ view_first,
                                                                          const float *__restrict__ x,
                                                                          double *__restrict__ acc)
{
    using T = FpTile<KW>;
    constexpr int W = T::W, G = T::G;
    extern __shared__ __align__(16) double fp_shared[];
    double(*s_x)[32] = reinterpret_cast<double(*)[32]>(fp_shared);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // column i's weights of this warp's view, then its number of entries
    double(*s_w)[W + 1] = reinterpret_cast<double(*)[W + 1]>(fp_shared + T::cols * 32) + warp * T::cols;
    const int nxy = g.N_x * g.N_y;
    const int n_chunks = (g.N_t + kRowChunk - 1) / kRowChunk;
    const int tiles_x = (g.N_x + T::TX - 1) / T::TX, tiles_y = (g.N_y + T::TY - 1) / T::TY;
    long long b = blockIdx.x;
    const int ch = (int)(b % n_chunks);
    b /= n_chunks;
    const int tx = (int)(b % tiles_x);
    b /= tiles_x;
    const int ty = (int)(b % tiles_y);
    const int f = (int)(b / tiles_y);
    const int t = ch * kRowChunk + lane;  // this lane's detector row
    const bool row_ok = t < g.N_t;
    for (int i = warp; i < T::cols; i += kFpWarps) {
        const int j = ty * T::TY + i / T::TX, k = tx * T::TX + i % T::TX;
        const bool in = j < g.N_y && k < g.N_x;
        s_x[i][lane] =
            (in && row_ok) ? (double)__ldg(x + ((size_t)f * nxy + (size_t)j * g.N_x + k) * g.N_z + t / g.z_overlap) : 0.0;
    }
    __syncthreads();
    // bit h of active: this lane's column of group h has a nonzero voxel
    unsigned active = 0;
    for (int i = 0; i < T::cols; i++)
        if (__any_sync(0xffffffffu, s_x[i][lane] != 0.0) && (i & 31) == lane) active |= 1u << (i >> 5);
    if (!__any_sync(0xffffffffu, active != 0)) return;
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const uint32_t *rec[G];
#pragma unroll
    for (int h = 0; h < G; h++) {
        const int i = h * 32 + lane, j = ty * T::TY + i / T::TX, k = tx * T::TX + i % T::TX;
        rec[h] = table + ((size_t)fv0 * nxy + ((active >> h & 1) ? (size_t)j * g.N_x + k : 0) * nv) * g.rec_words;
    }
    // a pair of views' records: 32 contiguous bytes a lane at KW 1
    uint4 R[2][G][KW];
    auto load = [&](int pair) {
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int h = 0; h < G; h++)
#pragma unroll
                for (int k = 0; k < KW; k++) {
                    const int v = 2 * pair + e;
                    R[e][h][k] = v < nv && (active >> h & 1)
                                     ? __ldg(reinterpret_cast<const uint4 *>(rec[h] + (size_t)v * g.rec_words) + k)
                                     : make_uint4(0u, 0u, 0u, 0u);
                }
    };
    const int pairs = (nv + 1) / 2, step = kFpWarps * gridDim.y;
    const double *my_x = &s_x[0][lane];
    int pair = blockIdx.y * kFpWarps + warp;
    if (pair < pairs) load(pair);
    for (; pair < pairs; pair += step) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            int row[G], lo = 0x7FFFFFFF, hi = -1;
#pragma unroll
            for (int h = 0; h < G; h++) {
                const uint32_t *words = &R[e][h][0].x;
                const int cnt = words[0] >> 24;
                row[h] = cnt ? (int)(words[0] & 0xFFFFFFu) : 0x7FFFFFFF;
                if (cnt) lo = min(lo, row[h]), hi = max(hi, row[h] + cnt - 1);
                double2 *dst = reinterpret_cast<double2 *>(s_w[h * 32 + lane]);
#pragma unroll
                for (int q = 0; q + 2 < W; q += 2)
                    dst[q / 2] = make_double2((double)__uint_as_float(words[1 + q]), (double)__uint_as_float(words[2 + q]));
                dst[W / 2] = make_double2((double)__uint_as_float(words[W]), __hiloint2double(0, cnt));
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            __syncwarp();
            if (e == 1 && pair + step < pairs) load(pair + step);  // in flight while this view is summed
            double a[W];
#pragma unroll
            for (int q = 0; q < W; q++) a[q] = 0.0;
            double *out = acc + (size_t)(hi < 0 ? 0 : lo) * g.N_t + t;
            for (int o = lo; o <= hi; o++, out += g.N_t) {
#pragma unroll
                for (int h = 0; h < G; h++) {
                    unsigned m = __ballot_sync(0xffffffffu, row[h] == o);
                    while (m) {
                        const int i = h * 32 + __ffs(m) - 1;
                        m &= m - 1;
                        const double xv = my_x[i * 32];
                        const double2 *src = reinterpret_cast<const double2 *>(s_w[i]);
                        double wt[W + 1];
#pragma unroll
                        for (int q = 0; q <= W; q += 2) {
                            const double2 u = src[q / 2];
                            wt[q] = u.x, wt[q + 1] = u.y;
                        }
                        const int cnt = __double2loint(wt[W]);
                        a[0] = fma(xv, wt[0], a[0]);
#pragma unroll
                        for (int q = 1; q < W; q++)
                            if (q < cnt) a[q] = fma(xv, wt[q], a[q]);
                    }
                }
                if (row_ok && a[0] != 0.0) atomicAdd(out, a[0]);
#pragma unroll
                for (int q = 0; q + 1 < W; q++) a[q] = a[q + 1];
                a[W - 1] = 0.0;
            }
            __syncwarp();  // the weights are read: the next view's may take their place
        }
    }
}

__global__ void finish_projection_kernel(size_t n, const double *__restrict__ acc, const float *__restrict__ y,
                                         float *__restrict__ out, const float *__restrict__ off, int nrt)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!y) {
            out[i] = (float)acc[i];
        } else {
            const float e = (float)((double)y[i] - acc[i]);
            out[i] = off ? e - off[i % nrt] : e;  // initErrorSinogam, XT_ICD_update.c:689
        }
    }
}

template <int KW>
static void launch_fp(const Geom &g, const uint32_t *d_table, const int32_t *d_view_first, const float *d_x, double *d_acc,
                      cudaStream_t st)
{
    using T = FpTile<KW>;
    const long long tiles = (long long)g.N_time * ((g.N_y + T::TY - 1) / T::TY) * ((g.N_x + T::TX - 1) / T::TX) *
                            ((g.N_t + kRowChunk - 1) / kRowChunk);
    // a frame's views over several CTAs where the tiles alone leave SMs idle
    const long long fill = 2 * 3 * 148, most = (g.N_p / g.N_time + 2 * kFpWarps - 1) / (2 * kFpWarps);
    const int parts = (int)std::max(1ll, std::min((fill + tiles - 1) / tiles, most));
    cudaFuncSetAttribute(forward_project_kernel<KW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::bytes);
    forward_project_kernel<KW>
        <<<dim3((unsigned)tiles, parts), kFpWarps * 32, T::bytes, st>>>(g, d_table, d_view_first, d_x, d_acc);
}

void launch_forward_project(const Geom &g, const uint32_t *d_table, const int32_t *d_view_first,
                            const float *d_x, const float *d_y, double *d_acc, float *d_out, cudaStream_t st,
                            const float *d_off)
{
    const size_t n = (size_t)g.N_p * g.N_r * g.N_t;
    cudaMemsetAsync(d_acc, 0, n * sizeof(double), st);
    if (g.rec_words == 4)
        launch_fp<1>(g, d_table, d_view_first, d_x, d_acc, st);
    else if (g.rec_words == 8)
        launch_fp<2>(g, d_table, d_view_first, d_x, d_acc, st);
    else
        launch_fp<3>(g, d_table, d_view_first, d_x, d_acc, st);
    finish_projection_kernel<<<148 * 8, 256, 0, st>>>(n, d_acc, d_y, d_out, d_off, g.N_r * g.N_t);
}

// VEC floats at p, zero where the predicate is off (then nothing is read)
template <int VEC>
__device__ __forceinline__ void load_rows(float (&v)[VEC], const float *p, bool on)
{
    if constexpr (VEC == 4)
        asm("{ .reg .pred q; setp.ne.s32 q, %5, 0; mov.f32 %0, 0f00000000; mov.f32 %1, 0f00000000; mov.f32 %2, 0f00000000; "
            "mov.f32 %3, 0f00000000; @q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4]; }"
            : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3])
            : "l"(p), "r"((int)on));
    else
        asm("{ .reg .pred q; setp.ne.s32 q, %3, 0; mov.f32 %0, 0f00000000; mov.f32 %1, 0f00000000; "
            "@q ld.global.nc.v2.f32 {%0, %1}, [%2]; }"
            : "=&f"(v[0]), "=&f"(v[1])
            : "l"(p), "r"((int)on));
}

// Back projection over one-word records (a header and up to 3 weights). A lane has
// VEC neighbouring detector rows, L = 32 / VEC lanes (fewer for a slab of fewer rows)
// cover a column's 32-row chunk and a warp has 32 / L neighbouring columns, a CTA a
// tile of them (8 x 4 at VEC 4): an instruction moves 512 B instead of 128, decoding a
// record costs each column a lane's share, and for one view the tile's entries fall
// on a few channels, which stay in L1. Twelve products (four views' entries) are
// summed in FP32, these sums in FP64. VEC 4 where the rows are a multiple of 4
// (16-byte loads), else 2 (the row counts are even). What bounds it: issue (59 % busy) and the
// latency of the rows' loads (L1, 78 % hits) at 24 warps an SM; 256 x 256 x 32 x 8 voxels, 1024
// views: 1.26 ms; a row a lane and a column a warp 2.79, four views of one column a
// warp 2.12 (its rows don't stay in L1), two or four CTAs an SM 1.40 and 1.58, the
// next records not loaded ahead 1.30.
template <int VEC>
__global__ void __launch_bounds__(256, 3) back_project_kernel(Geom g, int L, int cx, int cy, const uint4 *__restrict__ table,
                                                              const int32_t *__restrict__ view_first,
                                                              const float *__restrict__ sino, float *__restrict__ out)
{
    const int nxy = g.N_x * g.N_y;
    const int n_chunks = (g.N_t + kRowChunk - 1) / kRowChunk;
    const int tiles_x = (g.N_x + 4 * cx - 1) / (4 * cx), tiles_y = (g.N_y + 2 * cy - 1) / (2 * cy);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, own_col = lane / L;
    unsigned b = blockIdx.x;
    const int ch = (int)(b % n_chunks);
    b /= n_chunks;
    const int k = (int)(b % tiles_x) * 4 * cx + (warp & 3) * cx + own_col % cx;
    b /= tiles_x;
    const int j = (int)(b % tiles_y) * 2 * cy + (warp >> 2) * cy + own_col / cx;
    const int f = (int)(b / tiles_y);
    const int t = ch * kRowChunk + (lane & (L - 1)) * VEC;  // this lane's first detector row
    const bool ok = t < g.N_t && j < g.N_y && k < g.N_x;
    const int c = ok ? j * g.N_x + k : 0;
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const uint4 *rec = table + (size_t)fv0 * nxy + (size_t)c * nv;
    constexpr int U = 4;
    double acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; i++) acc[i] = 0.0;
    uint4 R[U], next[U];
#pragma unroll
    for (int u = 0; u < U; u++) next[u] = ok && u < nv ? __ldg(rec + u) : make_uint4(0, 0, 0, 0);
    for (int v0 = 0; v0 < nv; v0 += U) {
        // the next records are in flight while these views' rows are read
#pragma unroll
        for (int u = 0; u < U; u++) {
            R[u] = next[u];
            next[u] = ok && v0 + U + u < nv ? __ldg(rec + v0 + U + u) : make_uint4(0, 0, 0, 0);
        }
        float s[U][3][VEC];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int cnt = R[u].x >> 24;
            const float *p = sino + (size_t)(R[u].x & 0xFFFFFFu) * g.N_t + t;
#pragma unroll
            for (int q = 0; q < 3; q++) load_rows<VEC>(s[u][q], p + (size_t)q * g.N_t, q < cnt);
        }
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            float part = 0.0f;
#pragma unroll
            for (int u = 0; u < U; u++)
                part += __uint_as_float(R[u].y) * s[u][0][i] + __uint_as_float(R[u].z) * s[u][1][i] +
                        __uint_as_float(R[u].w) * s[u][2][i];
            acc[i] += (double)part;
        }
    }
    // z_overlap rows make a slice: first those of this lane, then its neighbours'
    const int zo = g.z_overlap, own = min(zo, VEC);
#pragma unroll
    for (int n = 1; n < VEC; n *= 2)
        if (n < own)
#pragma unroll
            for (int i = 0; i + n < VEC; i += 2 * n) acc[i] += acc[i + n];
    for (int off = 1; off < zo / VEC; off <<= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    if (ok && t % zo < VEC) {
        float *o = out + ((size_t)f * nxy + c) * g.N_z + t / zo;
#pragma unroll
        for (int i = 0; i < VEC; i++)
            if (i % own == 0) o[i / own] = (float)acc[i];
    }
}

// Back projection over longer records (coarse voxel scales): lane = detector row, one
// warp per column and chunk.
__global__ void back_project_wide_kernel(Geom g, const uint32_t *__restrict__ table,
                                         const int32_t *__restrict__ view_first, const float *__restrict__ sino,
                                         float *__restrict__ out)
{
    const int nxy = g.N_x * g.N_y;
    const int n_chunks = (g.N_t + kRowChunk - 1) / kRowChunk;
    const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= (long long)g.N_time * nxy * n_chunks) return;
    const int ch = (int)(gw % n_chunks);
    const long long fc = gw / n_chunks;
    const int f = (int)(fc / nxy), c = (int)(fc - (long long)f * nxy);
    const int t = ch * kRowChunk + lane;  // this lane's detector row
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const uint32_t *rec = table + ((size_t)fv0 * nxy + (size_t)c * nv) * g.rec_words;
    double acc = 0.0;
    if (t < g.N_t) {
        for (int v = 0; v < nv; v++, rec += g.rec_words) {
            const uint32_t hdr = __ldg(rec);
            const int cnt = hdr >> 24, row = hdr & 0xFFFFFF;
            for (int q = 0; q < cnt; q++) {
                const double a = (double)__uint_as_float(__ldg(rec + 1 + q));
                acc += a * (double)__ldg(sino + ((size_t)row + q) * g.N_t + t);
            }
        }
    }
    // rows of one voxel slice are z_overlap consecutive lanes (32 is a multiple of z_overlap)
    for (int off = 1; off < g.z_overlap; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (t < g.N_t && t % g.z_overlap == 0)
        out[((size_t)f * nxy + c) * g.N_z + t / g.z_overlap] = (float)acc;
}

// Back projection over z scales that do not divide a chunk of rows (no power of two, or
// above 32): lane = slice, which adds up its own z_overlap rows; one warp per column and
// 32 slices.
__global__ void back_project_slices_kernel(Geom g, const uint32_t *__restrict__ table,
                                           const int32_t *__restrict__ view_first, const float *__restrict__ sino,
                                           float *__restrict__ out)
{
    const int nxy = g.N_x * g.N_y;
    const int n_chunks = (g.N_z + 31) / 32;
    const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (gw >= (long long)g.N_time * nxy * n_chunks) return;
    const int z = (int)(gw % n_chunks) * 32 + (threadIdx.x & 31);
    if (z >= g.N_z) return;
    const long long fc = gw / n_chunks;
    const int f = (int)(fc / nxy), c = (int)(fc - (long long)f * nxy);
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const uint32_t *rec = table + ((size_t)fv0 * nxy + (size_t)c * nv) * g.rec_words;
    double acc = 0.0;
    for (int v = 0; v < nv; v++, rec += g.rec_words) {
        const uint32_t hdr = __ldg(rec);
        const int cnt = hdr >> 24;
        const float *p = sino + (size_t)(hdr & 0xFFFFFF) * g.N_t + (size_t)z * g.z_overlap;
        for (int q = 0; q < cnt; q++, p += g.N_t) {
            const double a = (double)__uint_as_float(__ldg(rec + 1 + q));
            for (int r = 0; r < g.z_overlap; r++) acc += a * (double)__ldg(p + r);
        }
    }
    out[((size_t)f * nxy + c) * g.N_z + z] = (float)acc;
}

void launch_back_project(const Geom &g, const uint32_t *d_table, const int32_t *d_view_first,
                         const float *d_sino, float *d_x, cudaStream_t st)
{
    const int chunks = (g.N_t + kRowChunk - 1) / kRowChunk;
    if (kRowChunk % g.z_overlap) {
        const long long warps = (long long)g.N_time * g.N_x * g.N_y * ((g.N_z + 31) / 32);
        back_project_slices_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(g, d_table, d_view_first, d_sino, d_x);
        return;
    }
    if (g.rec_words != 4) {
        const long long warps = (long long)g.N_time * g.N_x * g.N_y * chunks;
        back_project_wide_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(g, d_table, d_view_first, d_sino, d_x);
        return;
    }
    const uint4 *table = reinterpret_cast<const uint4 *>(d_table);
    const int vec = g.N_t % 4 == 0 ? 4 : 2;
    int L = 1, cx = 1, cy = 1;
    while (L * vec < std::min(g.N_t, kRowChunk)) L <<= 1;
    while (cx * cy * L < 32) (cx > cy ? cy : cx) <<= 1;
    const long long blocks =
        (long long)g.N_time * ((g.N_x + 4 * cx - 1) / (4 * cx)) * ((g.N_y + 2 * cy - 1) / (2 * cy)) * chunks;
    if (vec == 4)
        back_project_kernel<4><<<(unsigned)blocks, 256, 0, st>>>(g, L, cx, cy, table, d_view_first, d_sino, d_x);
    else
        back_project_kernel<2><<<(unsigned)blocks, 256, 0, st>>>(g, L, cx, cy, table, d_view_first, d_sino, d_x);
}

}  // namespace mbirgpu
