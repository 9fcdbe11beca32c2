// Non-homogeneous ICD voxel-line selection on the GPU.
//
// Replaces VSC_based_Voxel_Line_Select and ComputeVSC (MBIR_4D/XT_NHICD.c:
// 128-216). Per frame: the per-column update magnitude of the latest visit
// (sum over z of |x_new - x_old|, MagUpdateMap, XT_VoxUpdate.c:158,265) is
// filtered with the reference's 5x5 Hamming window (FP64 sum, stored as
// float like filtMagUpdateMap); the threshold is the (N - k)-th smallest
// filtered value over all N = N_y N_x columns (RandomizedSelect's order
// statistic), found here by an exact 4-digit radix select on the float bit
// patterns (non-negative floats order like their bits) by a cluster of CTAs
// per frame; the selected columns
// are those strictly above it -- the k largest -- that lie inside the mask
// (the reference also picks unmasked columns near the edge but its update
// skips them, XT_VoxUpdate.c:168).
#include <algorithm>

#include "mbir_internal.h"

namespace mbirgpu {

namespace {

__constant__ double c_hamming[5][5] = {{0.0064, 0.0432, 0.0800, 0.0432, 0.0064},
                                       {0.0432, 0.2916, 0.5400, 0.2916, 0.0432},
                                       {0.0800, 0.5400, 1.0000, 0.5400, 0.0800},
                                       {0.0432, 0.2916, 0.5400, 0.2916, 0.0432},
                                       {0.0064, 0.0432, 0.0800, 0.0432, 0.0064}};

// filtered update magnitude of column (j, k): the reference's 5x5 window in its
// (p, q) order, FP64 without contraction, as the host
__device__ __forceinline__ float vsc_filter(const float *__restrict__ m, int j, int k, int NY, int NX)
{
    double acc = 0.0;
#pragma unroll
    for (int p = -2; p <= 2; p++) {
        const int jj = j + p;
        if (jj < 0 || jj >= NY) continue;
#pragma unroll
        for (int q = -2; q <= 2; q++) {
            const int kk = k + q;
            if (kk < 0 || kk >= NX) continue;
            acc = __dadd_rn(acc, __dmul_rn(c_hamming[p + 2][q + 2], (double)m[jj * NX + kk]));
        }
    }
    return (float)acc;
}

// walk each phase's SVs in the sweep's own queue order (frames fastest, spread
// slots) and append the non-empty ones to their count's bucket
__global__ void __launch_bounds__(256) nh_scatter_kernel(int n_frames, int NY, int NX, int sv, int K, int perm, int per_phase,
                                                         const int *__restrict__ svcount, const int *__restrict__ hist,
                                                         int *__restrict__ cursor, uint32_t *__restrict__ items,
                                                         int *__restrict__ n_items)
{
    // the bucket of c columns starts after the buckets of more: every CTA adds
    // up its phase's histogram (blockIdx.y: the phase)
    __shared__ int s_off[257];
    const int p = blockIdx.y;
    const int nsx = (NX + sv - 1) / sv, nsy = (NY + sv - 1) / sv, maxc = sv * sv, KK = K * K;
    for (int c = threadIdx.x; c <= maxc; c += blockDim.x) s_off[c] = hist[p * (maxc + 1) + c];
    __syncthreads();
    if (threadIdx.x == 0) {
        int o = 0;
        for (int c = maxc; c >= 1; c--) {
            const int h = s_off[c];
            s_off[c] = o;
            o += h;
        }
        if (blockIdx.x == 0) n_items[p] = o;
    }
    __syncthreads();
    const int hx = (nsx + K - 1) / K, slots = hx * ((nsy + K - 1) / K);
    const int n = n_frames * slots;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int f = q % n_frames;
        const int rem = (int)((long long)(q / n_frames) * perm % slots);
        const int color = (p + f) % KK;
        const int sx = K * (rem % hx) + color % K, sy = K * (rem / hx) + color / K;
        if (sx >= nsx || sy >= nsy) continue;
        const int cnt = svcount[((size_t)f * nsy + sy) * nsx + sx];
        if (!cnt) continue;
        const int pos = atomicAdd(&cursor[p * (maxc + 1) + cnt], 1);
        items[(size_t)p * per_phase + s_off[cnt] + pos] = ((uint32_t)f << 22) | ((uint32_t)sy << 11) | (uint32_t)sx;
    }
}

// The selection of one pass, one cluster of kSelCtas CTAs per frame: the filtered
// map; its threshold, the (k + 1)-th largest value, by radix select over the float
// bit patterns, eight bits a round (each CTA's histogram of the keys that match
// the digits so far in its shared memory, added up over the cluster through
// distributed shared memory, so every CTA finds the same digit); sel = mask && key
// > threshold; and, when svcount is given, the selected columns of every
// super-voxel with a histogram per (phase, count). One launch: as eleven (filter,
// four histogram / pick pairs, ...) a pass's selection took about 65 us, most of it
// launches and one thread scanning 256 bins. Images beyond 65,536 columns are filtered by
// a launch of their own first: 27 us for 512 x 512 columns, 69 for 1024 x 1024, 234 for
// 2048 x 2048 (filtered by the eight SMs of the cluster 80, 294 and 1,102; as eleven
// launches 72, 124 and 358).
constexpr int kSelCtas = 8, kSelThreads = 1024;
constexpr int kSelKeys = 8;  // keys a thread keeps in registers (images up to 256 x 256 entirely)

// The filtered map of a larger image, by the whole GPU: eight SMs a frame take longer over
// the filter than over the rest of the selection.
__global__ void __launch_bounds__(256) nh_filter_kernel(int n_frames, int NY, int NX, const float *__restrict__ mag,
                                                        float *__restrict__ filt)
{
    const int nxy = NX * NY;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)n_frames * nxy;
         i += (long long)gridDim.x * blockDim.x) {
        const int f = (int)(i / nxy), c = (int)(i - (long long)f * nxy);
        filt[i] = vsc_filter(mag + (size_t)f * nxy, c / NX, c % NX, NY, NX);
    }
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned remote_load(const unsigned *p, unsigned rank)
{
    unsigned a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

__global__ void __cluster_dims__(kSelCtas, 1, 1) __launch_bounds__(kSelThreads)
    nh_select_kernel(int NY, int NX, int k, const float *__restrict__ mag, const uint8_t *__restrict__ mask,
                     const float *__restrict__ filt, uint8_t *__restrict__ sel, int sv, int K, int *__restrict__ svcount,
                     int *__restrict__ hist_out)
{
    __shared__ unsigned s_hist[256], s_sum[256];
    __shared__ unsigned s_digit, s_above;
    const int f = blockIdx.x / kSelCtas, rank = blockIdx.x % kSelCtas;
    const int nxy = NX * NY, first = rank * kSelThreads + threadIdx.x, stride = kSelCtas * kSelThreads;
    const float *m = mag + (size_t)f * nxy;
    const float *fm = filt + (size_t)f * nxy;
    uint8_t *sm = sel + (size_t)f * nxy;
    unsigned key[kSelKeys];
    const int rest = first + kSelKeys * stride;  // columns past those: read from the map (nh_filter_kernel) each time
    const bool mapped = nxy > kSelKeys * stride;
#pragma unroll
    for (int i = 0; i < kSelKeys; i++) {
        const int c = first + i * stride;
        key[i] = c >= nxy ? 0u : __float_as_uint(mapped ? fm[c] : vsc_filter(m, c / NX, c % NX, NY, NX));
    }
    unsigned prefix = 0, pmask = 0, need = (unsigned)k + 1;
    bool found = true;
    for (int shift = 24; shift >= 0 && found; shift -= 8) {  // uniform over the cluster
        for (int b = threadIdx.x; b < 256; b += kSelThreads) s_hist[b] = 0u;
        __syncthreads();
        auto count = [&](unsigned u) {
            if ((u & pmask) == prefix) atomicAdd(&s_hist[(u >> shift) & 255u], 1u);
        };
#pragma unroll
        for (int i = 0; i < kSelKeys; i++)
            if (first + i * stride < nxy) count(key[i]);
#pragma unroll 8
        for (int c = rest; c < nxy; c += stride) count(__float_as_uint(fm[c]));
        cluster_sync();
        if (threadIdx.x < 256) {
            unsigned t = 0;
            for (unsigned r = 0; r < kSelCtas; r++) t += remote_load(&s_hist[threadIdx.x], r);
            s_sum[threadIdx.x] = t;
        }
        __syncthreads();
        // the digit at which the count from the top reaches the rank: lane l of warp 0
        // holds digits 255 - 8 l .. 248 - 8 l
        if (threadIdx.x < 32) {
            unsigned h[8], t = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) t += h[i] = s_sum[255 - 8 * threadIdx.x - i];
            unsigned incl = t;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned up = __shfl_up_sync(0xffffffffu, incl, o);
                if (threadIdx.x >= o) incl += up;
            }
            const unsigned any = __ballot_sync(0xffffffffu, incl >= need);
            if (any == 0) {
                if (threadIdx.x == 0) s_digit = 256u;  // fewer keys than the rank: all are above the threshold
            } else if ((int)threadIdx.x == __ffs(any) - 1) {
                unsigned cum = incl - t;
                int i = 0;
                while (cum + h[i] < need) cum += h[i++];
                s_digit = 255u - 8u * threadIdx.x - (unsigned)i;
                s_above = cum;
            }
        }
        __syncthreads();
        found = s_digit < 256u;
        if (found) {
            prefix |= s_digit << shift;
            pmask |= 0xFFu << shift;
            need -= s_above;
        }
        cluster_sync();  // every CTA has read this round's histograms
    }
#pragma unroll
    for (int i = 0; i < kSelKeys; i++) {
        const int c = first + i * stride;
        if (c < nxy) sm[c] = (uint8_t)(k > 0 && mask[c] && (!found || key[i] > prefix));
    }
#pragma unroll 8
    for (int c = rest; c < nxy; c += stride)
        sm[c] = (uint8_t)(k > 0 && mask[c] && (!found || __float_as_uint(fm[c]) > prefix));
    if (!svcount) return;
    cluster_sync();  // the frame's selection is complete
    const int nsx = (NX + sv - 1) / sv, nsy = (NY + sv - 1) / sv, maxc = sv * sv;
    for (int i = first; i < nsx * nsy; i += stride) {
        const int sy = i / nsx, sx = i - sy * nsx;
        int cnt = 0;
        for (int a = 0; a < sv && sy * sv + a < NY; a++)
            for (int b = 0; b < sv && sx * sv + b < NX; b++) cnt += __ldcg(sm + (sy * sv + a) * NX + sx * sv + b) != 0;
        svcount[(size_t)f * nsx * nsy + i] = cnt;
        if (cnt) {
            const int color = (sy % K) * K + sx % K;
            const int phase = ((color - f) % (K * K) + K * K) % (K * K);
            atomicAdd(&hist_out[phase * (maxc + 1) + cnt], 1);
        }
    }
}

}  // namespace

int nh_items_per_phase(int n_frames, int N_y, int N_x, int sv, int K)
{
    return n_frames * sv_slots(N_x, N_y, sv, K);
}

// [svcount | hist | cursor]
size_t nh_items_scratch_ints(int n_frames, int N_y, int N_x, int sv, int K)
{
    const size_t nsv = (size_t)((N_x + sv - 1) / sv) * ((N_y + sv - 1) / sv);
    return (size_t)n_frames * nsv + 2 * (size_t)K * K * (sv * sv + 1);
}

bool nh_items_supported(int n_frames, int N_y, int N_x, int sv)
{
    return n_frames <= 1024 && (N_x + sv - 1) / sv <= 2048 && (N_y + sv - 1) / sv <= 2048;
}

// Returns the kernels launched.
static int filter_large(int n_frames, int N_y, int N_x, const float *d_mag, float *d_filt, cudaStream_t st)
{
    const long long n = (long long)n_frames * N_y * N_x;
    if ((long long)N_y * N_x <= (long long)kSelKeys * kSelCtas * kSelThreads) return 0;
    nh_filter_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 148 * 8), 256, 0, st>>>(n_frames, N_y, N_x, d_mag, d_filt);
    return 1;
}

int launch_nh_select(int n_frames, int N_y, int N_x, const float *d_mag, const uint8_t *d_mask, int k,
                     float *d_filt, uint8_t *d_sel, cudaStream_t st)
{
    const int launched = filter_large(n_frames, N_y, N_x, d_mag, d_filt, st);
    nh_select_kernel<<<kSelCtas * n_frames, kSelThreads, 0, st>>>(N_y, N_x, k, d_mag, d_mask, d_filt, d_sel, 1, 1, nullptr,
                                                                 nullptr);
    return launched + 1;
}

int launch_nh_select_items(int n_frames, int N_y, int N_x, const float *d_mag, const uint8_t *d_mask, int k,
                           float *d_filt, uint8_t *d_sel, int sv, int K, uint32_t *d_items, int *d_n_items, int *d_scratch,
                           cudaStream_t st)
{
    const int nsx = (N_x + sv - 1) / sv, nsy = (N_y + sv - 1) / sv, maxc = sv * sv, KK = K * K;
    const size_t nsv = (size_t)n_frames * nsx * nsy, hsz = (size_t)KK * (maxc + 1);
    int *svcount = d_scratch, *hist = d_scratch + nsv, *cursor = hist + hsz;
    cudaMemsetAsync(hist, 0, 2 * hsz * sizeof(int), st);
    const int launched = filter_large(n_frames, N_y, N_x, d_mag, d_filt, st);
    nh_select_kernel<<<kSelCtas * n_frames, kSelThreads, 0, st>>>(N_y, N_x, k, d_mag, d_mask, d_filt, d_sel, sv, K, svcount,
                                                                 hist);
    const int per_phase = nh_items_per_phase(n_frames, N_y, N_x, sv, K);
    nh_scatter_kernel<<<dim3((per_phase + 255) / 256, KK), 256, 0, st>>>(
        n_frames, N_y, N_x, sv, K, spread_multiplier(sv_slots(N_x, N_y, sv, K)), per_phase, svcount, hist, cursor, d_items,
        d_n_items);
    return launched + 2;
}

}  // namespace mbirgpu
