// FP64 MAP cost (replaces computeCost, MBIR_4D/XT_ICD_update.c:185-318).
//
// Data term: 1/2 sum w e^2 where |e sqrt(w)| < T, else the generalised-Huber
// branch 2 delta T |e sqrt(w)| + T^2 (1 - 2 delta) (XT_ICD_update.c:192-204);
// the test is made as e^2 w < T^2.
// Prior term: for every voxel the 13 causal spatial pairs (+x; the three +y
// pairs of its slice; the nine pairs of the next slice) and the +t pair, each
// filter weight times the qGGMRF potential |d|^q / sigma^q / (c + |d|^(q-p) /
// sigma^(q-p)) (XT_ICD_update.c:82-90, 206-298). Neighbour differences are
// taken in float as the reference's float - float. The log-variance term is
// zero (variance estimate 1).
//
// Deterministic: every block writes its partial sums, then one block adds the
// partials in a fixed order (thread by thread, then its tree).
#include "mbir_internal.h"

namespace mbirgpu {

namespace {
constexpr int kCostThreads = 256;
constexpr int kCostBlocks = 148 * 6;  // two waves at three blocks an SM
}

int cost_partials_needed(const Geom &) { return 2 * kCostBlocks; }

// The qGGMRF potential |d|^q / sq / (c + |d|^(q-p) / sqp) in FP64, 14 times a voxel,
// is the time of this kernel. The powers of the float |d| come from a table-driven
// logarithm and exponential (Tang's method: an argument near a tabulated point, a
// short polynomial in the rest), the quotient from a cubic step (Halley's) on an
// approximate reciprocal, fused into the sum: about 28 FP64 instructions and 4
// table reads, as exact against the FP64 oracle as the library's functions. A
// voxel's 14 evaluations have no branch between them, so their chains overlap.
// 256 x 256 x 32 x 8 voxels and 512 MB of sinogram: library functions 1.53 ms; this
// form with a branch per difference 1.05; without 0.64 (80 registers, three blocks an
// SM; 64 registers spill, 0.71; 103 registers, two blocks, 0.78). Tables of 16 entries,
// whose reads never conflict, need longer polynomials: 1.24 against 1.05.
struct PowTables {
    double inv[128], lg[128];  // 1 / c_i and -log2 of it, c_i = 1 + (i + 1/2) / 128
    double e2[64];             // 2^(j / 64)
};

__device__ inline void fill_tables(PowTables &T)
{
    for (int i = threadIdx.x; i < 128; i += blockDim.x) {
        T.inv[i] = 1.0 / (1.0 + (i + 0.5) / 128.0);
        T.lg[i] = -log2(T.inv[i]);
    }
    for (int i = threadIdx.x; i < 64; i += blockDim.x) T.e2[i] = exp2(i / 64.0);
}

// log2 of a positive normal double
__device__ __forceinline__ double log2_of(double a, const PowTables &T)
{
    const int hi = __double2hiint(a), i = (hi >> 13) & 127;
    const double m = __hiloint2double((hi & 0xFFFFF) | 0x3FF00000, __double2loint(a));
    // the exponent as a double: 2^52 + 2^31 + e less 2^52 + 2^31
    const double e = __hiloint2double(0x43300000, (int)(0x80000000u + (unsigned)((hi >> 20) - 1023))) - 4503601774854144.0;
    const double r = fma(m, T.inv[i], -1.0);  // |r| <= 2^-8
    // log2(1 + r) / r up to r^5
    constexpr double k = 1.4426950408889634;
    double p = fma(r, -k / 6, k / 5);
    p = fma(r, p, -k / 4);
    p = fma(r, p, k / 3);
    p = fma(r, p, -k / 2);
    p = fma(r, p, k);
    return fma(r, p, T.lg[i] + e);
}

// 2^y, |y| < 1000
__device__ __forceinline__ double exp2_of(double y, const PowTables &T)
{
    const double magic = 6755399441055744.0;  // 1.5 2^52: the sum's low bits are the rounded integer
    const double t = fma(y, 64.0, magic);
    const int n = __double2loint(t);
    const double f = fma(t - magic, -1.0 / 64, y);  // |f| <= 1 / 128
    constexpr double a = 0.69314718055994531;
    double p = fma(f, a * a * a * a * a / 120, a * a * a * a / 24);
    p = fma(f, p, a * a * a / 6);
    p = fma(f, p, a * a / 2);
    p = fma(f, p, a);
    const double e = T.e2[n & 63];
    const double v = fma(e, f * p, e);
    return __hiloint2double(__double2hiint(v) + ((n >> 6) << 20), __double2loint(v));
}

// The largest exponent whose powers stay in exp2_of's range: |d| is 2^-149 to 2^128.
constexpr double kMaxFastQ = 6.5;

// sum += |d|^q / (c + |d|^(q-p) / sqp), branch-free so that several run at once. A
// zero difference adds nothing; bad is set where the fast form does not hold (an
// infinite or NaN difference, a denominator outside 2^-100 .. 2^100; the caller sets it
// for exponents past kMaxFastQ).
__device__ __forceinline__ void add_potential(double &sum, bool &bad, float d, double q, double qmp, double inv_sqp,
                                              double c, const PowTables &T)
{
    const double ad = (double)fmaxf(fabsf(d), 1.0e-45f);
    const double lg = log2_of(ad, T);
    const double num = q == 2.0 ? ad * ad : exp2_of(q * lg, T);
    const double den = fma(exp2_of(qmp * lg, T), inv_sqp, c);
    bad |= (unsigned)(__double2hiint(den) >> 20) - 923u > 200u || !(fabsf(d) < INFINITY);
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(den));
    const double e = fma(-den, r, 1.0), n = d != 0.0f ? num * r : 0.0;  // num / den = n / (1 - e) = n (1 + e + e^2) to e^3
    sum = fma(n, fma(e, e, e), sum + n);
}

// the same by the library's functions
__device__ __noinline__ double plain_potential(float d, double q, double qmp, double inv_sqp, double c)
{
    if (d == 0.0f) return 0.0;
    const double ad = fabs((double)d), l = log(ad);
    return (q == 2.0 ? ad * ad : exp(q * l)) / (c + exp(qmp * l) * inv_sqp);
}

__device__ inline double block_sum(double v, double *sh)
{
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double s = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += sh[i];
    return s;  // valid in thread 0
}

// x is [N_time][N_y][N_x][N_z]
__global__ void __launch_bounds__(kCostThreads) cost_partials_kernel(Geom g, const float *__restrict__ err,
                                                                    const float *__restrict__ w,
                                                                    const float *__restrict__ x,
                                                                    double *__restrict__ partials)
{
    __shared__ double sh[kCostThreads / 32];
    __shared__ PowTables T;
    fill_tables(T);
    __syncthreads();
    const long long nsino = (long long)g.N_p * g.N_r * g.N_t;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    double data = 0;
    const double T2 = g.huber_T * g.huber_T;
    for (long long i = tid; i < nsino; i += stride) {
        // |e sqrt(w)| < T  <=>  e^2 w < T^2; the square root is only needed on the Huber branch
        const double e = (double)err[i], ww = (double)w[i];
        const double t2 = e * e * ww;
        if (t2 < T2) data += t2;
        else data += 2.0 * g.huber_delta * g.huber_T * sqrt(t2) + T2 * (1.0 - 2.0 * g.huber_delta);
    }
    const double qmp = g.q - g.p;
    const double inv_ssq = 1.0 / g.sigma_s_q, inv_ssqp = 1.0 / g.sigma_s_q_p;
    const double inv_stq = 1.0 / g.sigma_t_q, inv_stqp = 1.0 / g.sigma_t_q_p;
    const int NX = g.N_x, NY = g.N_y, NZ = g.N_z, NT = g.N_time;
    const int nxy = NX * NY;
    // a group of zp lanes per voxel column (zp a power of two, at most a warp),
    // lanes over its slices
    int zp = 1;
    while (zp < NZ && zp < 32) zp <<= 1;
    const int z_first = threadIdx.x & (zp - 1);
    const long long groups = stride / zp, ncol = (long long)NT * nxy;
    double prior = 0;
    for (long long col = tid / zp; col < ncol; col += groups) {
        const int f = (int)(col / nxy), c2 = (int)(col - (long long)f * nxy), j = c2 / NX, k = c2 - j * NX;
        const bool jm = j > 0, km = k > 0, jp = j + 1 < NY, kp = k + 1 < NX;
        const float *xc = x + (size_t)col * NZ;
        const ptrdiff_t dx = NZ, dy = (ptrdiff_t)NX * NZ;
        for (int z = z_first; z < NZ; z += zp) {
            const float c = xc[z];
            // half of the neighbours: 3 at distance 1, 6 at sqrt 2, 4 at sqrt 3, which
            // share a filter weight each, and the next frame's voxel; one outside
            // the volume has a difference of zero, which adds nothing
            const bool zp1 = z + 1 < NZ;
            float d[14];
            auto D = [&](bool in, ptrdiff_t off) { return in ? c - xc[z + (in ? off : 0)] : 0.0f; };
            d[0] = D(kp, dx), d[1] = D(jp, dy), d[2] = D(zp1, 1);
            d[3] = D(jp && km, dy - dx), d[4] = D(jp && kp, dy + dx);
            d[5] = D(zp1 && jm, 1 - dy), d[6] = D(zp1 && km, 1 - dx), d[7] = D(zp1 && kp, 1 + dx), d[8] = D(zp1 && jp, 1 + dy);
            d[9] = D(zp1 && jm && km, 1 - dy - dx), d[10] = D(zp1 && jm && kp, 1 - dy + dx);
            d[11] = D(zp1 && jp && km, 1 + dy - dx), d[12] = D(zp1 && jp && kp, 1 + dy + dx);
            d[13] = D(f + 1 < NT, (ptrdiff_t)nxy * NZ);
            bool any = false;
#pragma unroll
            for (int i = 0; i < 14; i++) any |= d[i] != 0.0f;
            if (!any) continue;
            double s[4] = {0, 0, 0, 0};
            bool bad = !(g.q <= kMaxFastQ);
#pragma unroll
            for (int i = 0; i < 14; i++)
                add_potential(s[i < 3 ? 0 : i < 9 ? 1 : i < 13 ? 2 : 3], bad, d[i], g.q, qmp, i < 13 ? inv_ssqp : inv_stqp,
                              i < 13 ? g.c_s : g.c_t, T);
            if (bad) {
#pragma unroll
                for (int i = 0; i < 4; i++) s[i] = 0;
#pragma unroll
                for (int i = 0; i < 14; i++)
                    s[i < 3 ? 0 : i < 9 ? 1 : i < 13 ? 2 : 3] +=
                        plain_potential(d[i], g.q, qmp, i < 13 ? inv_ssqp : inv_stqp, i < 13 ? g.c_s : g.c_t);
            }
            prior += (g.spatial_filter[9 + 3 + 2] * s[0] + g.spatial_filter[9 + 6 + 2] * s[1] + g.spatial_filter[18 + 6 + 2] * s[2]) * inv_ssq +
                     g.time_filter * inv_stq * s[3];
        }
    }
    const double ds = block_sum(data, sh);
    const double ps = block_sum(prior, sh);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = ds;
        partials[gridDim.x + blockIdx.x] = ps;
    }
}

// the blocks' partial sums in a fixed order: thread t adds partials t, t + 256, ...,
// then the block's tree (one thread adding all of them took 61 us)
__global__ void __launch_bounds__(kCostThreads) cost_finish_kernel(const double *__restrict__ partials, int nblocks,
                                                                  double *__restrict__ out)
{
    __shared__ double sh[kCostThreads / 32];
    double d = 0, p = 0;
    for (int i = threadIdx.x; i < nblocks; i += kCostThreads) {
        d += partials[i];
        p += partials[nblocks + i];
    }
    const double ds = block_sum(d, sh), ps = block_sum(p, sh);
    if (threadIdx.x == 0) {
        out[0] = ds / 2.0;
        out[1] = ps;
    }
}

void launch_cost(const Geom &g, const float *d_err, const float *d_w, const float *d_x, double *d_partials,
                 int n_partials, double *d_out, cudaStream_t st)
{
    const int blocks = n_partials / 2;
    cost_partials_kernel<<<blocks, kCostThreads, 0, st>>>(g, d_err, d_w, d_x, d_partials);
    cost_finish_kernel<<<1, kCostThreads, 0, st>>>(d_partials, blocks, d_out);
}

}  // namespace mbirgpu
