// Super-voxel parallel ICD sweep (one colour phase per launch).
//
// Replaces the voxel loop of updateVoxelsTimeSlices / updateVoxels_Atten /
// compute_voxel_update_Atten (MBIR_4D/XT_ICD_update.c:932-1092,
// XT_VoxUpdate.c:45-283) and the surrogate solve CE_FunctionalSubstitution
// (XT_ICD_update.c:133-182).
//
// Schedule. The image plane is tiled into super-voxels (SVs) of sv x sv voxel
// columns; with K x K colours (K = 2 or 4) an SV's colour is
// (sv_y mod K) K + (sv_x mod K). Phase p updates, in frame f, the SVs of
// colour (p + f) mod K^2: no two SVs updated at once share a prior neighbour,
// and a voxel and its temporal neighbours (same column, frames f +- 1) are
// never updated at once -- the GPU counterpart of the reference's z-block /
// frame checkerboard (XT_ICD_update.c:964-1046). Frames use disjoint views,
// so different frames never share sinogram entries; concurrent SVs of one
// frame can share entries along a ray, and their error sinogram updates are
// atomic adds (how many may run at once is bounded by sv_max_concurrent).
//
// A grid of persistent CTAs (as many as fit on the GPU) drains a queue of the
// phase's SVs, frames fastest and SV slots in a spread order (queue index x
// perm mod slots), so the SVs in flight are far apart; a CTA owns one SV at a
// time and visits its voxel columns one
// after another in a seeded random order (the counterpart of
// randomly_select_x_y, XT_ICD_update.c:499-531). For one column all warps
// cooperate, with two CTA barriers per column:
//   1. neighbourhood: the 8 in-plane neighbour columns and the 2 temporal
//      neighbours are split over the warps; each lane owns one slice z and
//      accumulates the qGGMRF surrogate terms b = w rho'(d)/d of those
//      neighbours (XT_ICD_update.c:140-172), read from a tile of the SV and its
//      surroundings in shared memory where it fits; whether any slice escapes zero
//      skipping (XT_VoxUpdate.c:238-261) is decided from the same reads;
//   2. theta: the column's A entries lie in lists in shared memory, one per warp
//      and view group, unpacked from the records while the column before was
//      solved; a lane owns VEC consecutive detector rows and accumulates theta1 =
//      -sum a w e and theta2 = sum a^2 w over its list (a = A value x delta_t,
//      XT_VoxUpdate.c:56-85) in packed FP32 arithmetic, a batch of up to 8
//      entries' e and w in flight at once;
//   3. solve: warp 0 sums the partials, then updates even slices and odd
//      slices in turn (their only mutual coupling is the in-column z +- 1
//      prior pair), x <- V + alpha (u - V);
//   4. apply: e[view][r][t] -= a dx(slice of t) with vector reductions.
// All arithmetic is FP32; the host refreshes e in FP64 periodically.
#include <mutex>
#include <vector>

#include "mbir_internal.h"

namespace mbirgpu {

namespace {

constexpr int kMaxWarps = 8;
constexpr int kMaxSvCols = 256;  // sv <= 16
constexpr float kMinNormal = 1.17549435e-38f;  // 2^-126
constexpr float kHuberMaxZ = 1e30f, kHuberMinW = 1e-12f, kHuberMaxW = 1e12f;  // the short linear weight's range

__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Surrogate weight rho'(d)/d of the qGGMRF potential
// |d|^(q-p) ... (derivative per XT_ICD_update.c:92-118; value at d = 0 per
// :119-128): |d|^(q-2) (q - (q-p) t1 / t3) / (t3 sq), t1 = |d|^(q-p) / sqp,
// t3 = c + t1. The weight is evaluated ~28 times per voxel update, so it uses
// the hardware base-2 logarithm / exponential (one logarithm for both powers)
// and reciprocal: FP32 arithmetic whose rounding the FP64 MAP cost, by which
// the method's result is measured, does not see.
__device__ __forceinline__ float lg2_hw(float x)
{
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float ex2_hw(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_hw(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// N weights times their filter coefficients f (which carry the 1 / sq), side by
// side and without branches, so that the N chains of about 130 cycles run in
// each other's shadow. isqp = 1 / sqp; at d = 0 the weight is q / (sq c), and below
// 2^-126, which the logarithm takes for zero (an infinite |d|^(q-2) at q < 2), too.
template <int N>
__device__ __forceinline__ void qg_coef(const float (&d)[N], const float (&f)[N], float q, float qmp, float isqp,
                                        float c, float qoc, float (&cf)[N])
{
    float l[N];
#pragma unroll
    for (int i = 0; i < N; i++) l[i] = lg2_hw(fabsf(d[i]));
#pragma unroll
    for (int i = 0; i < N; i++) {
        const float t1 = ex2_hw(qmp * l[i]) * isqp;
        const float rt3 = rcp_hw(c + t1);
        cf[i] = (q - qmp * (t1 * rt3)) * rt3;
    }
    if (q != 2.0f) {
#pragma unroll
        for (int i = 0; i < N; i++) cf[i] *= ex2_hw((q - 2.0f) * l[i]);
    }
#pragma unroll
    for (int i = 0; i < N; i++) cf[i] = f[i] * (fabsf(d[i]) < kMinNormal ? qoc : cf[i]);
}

// The one arrival of a copy's mbarrier phase, and the bytes the phase waits for.
__device__ __forceinline__ void expect_bytes(unsigned long long *bar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
                 "r"(bytes)
                 : "memory");
}
// One TMA bulk copy into shared memory (16-byte aligned on both sides, a multiple
// of 16 bytes), issued by one thread; completes on the mbarrier.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar))
                 : "memory");
}

// The voxel values a super-voxel's updates read, by bulk copies into shared
// memory: three planes of (sv + 2)^2 columns -- the SV and its in-plane
// neighbours in its frame, then the SV's columns in frames f - 1 and f + 1 at
// the same places of their planes, so that every neighbour of a column sits at a
// fixed offset from it. A plane's row is contiguous in x ([y][x][z]); cells
// outside the image or the frames are left alone (never read). Called by one
// warp; N_z is a multiple of 4, so every row starts on 16 bytes and is a multiple
// of 16 bytes long. `more`: bytes of a further copy on the same mbarrier phase.
// No other CTA of the launch writes these columns (same-colour SVs share no
// neighbour, and frames f +- 1 are on other colours).
__device__ __forceinline__ void stage_tile(float *tile, const float *x, const Geom &g, int f, int sx, int sy, int sv,
                                           int more, unsigned long long *bar)
{
    const int lane = threadIdx.x & 31, TW = sv + 2, NX = g.N_x, NY = g.N_y, NZ = g.N_z;
    const size_t nxy = (size_t)NX * NY;
    const int j0 = sy * sv, k0 = sx * sv;
    const int ka = max(k0 - 1, 0), kb = min(k0 + sv + 1, NX), ja = max(j0 - 1, 0), jb = min(j0 + sv + 1, NY);
    const int ke = min(k0 + sv, NX), je = min(j0 + sv, NY);
    const int frames = (f > 0) + (f + 1 < g.N_time);
    if (lane == 0) expect_bytes(bar, 4 * NZ * ((jb - ja) * (kb - ka) + frames * (je - j0) * (ke - k0)) + more);
    __syncwarp();
    for (int r = lane; r < TW + 2 * sv; r += 32) {
        if (r < TW) {
            const int j = j0 - 1 + r;
            if (j >= 0 && j < NY)
                bulk_copy(tile + (r * TW + (ka - k0 + 1)) * NZ, x + ((size_t)f * nxy + (size_t)j * NX + ka) * NZ,
                          4u * (unsigned)((kb - ka) * NZ), bar);
        } else {
            const int p = r - TW < sv ? 1 : 2, row = r - TW - (p - 1) * sv, ff = p == 1 ? f - 1 : f + 1, j = j0 + row;
            if (ff >= 0 && ff < g.N_time && j < NY)
                bulk_copy(tile + ((p * TW + row + 1) * TW + 1) * NZ, x + ((size_t)ff * nxy + (size_t)j * NX + k0) * NZ,
                          4u * (unsigned)((ke - k0) * NZ), bar);
        }
    }
}

__device__ __forceinline__ bool try_parity(unsigned long long *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(ok)
        : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait (about 2 s of clock64) for phase `parity` of mbarrier `bar`;
// returns false if it ran out.
__device__ __forceinline__ bool wait_parity_bounded(unsigned long long *bar, uint32_t parity)
{
    if (try_parity(bar, parity)) return true;  // the usual case: the copy landed a column ago
    const long long t0 = clock64();
    while (!try_parity(bar, parity))
        if (clock64() - t0 > 4000000000LL) return false;
    return true;
}

// Wait for buffer b's copy: the n-th copy into a buffer completes the mbarrier's
// phase n, so the parity of the wait is the count of earlier copies into that
// buffer (bit b of `phases`, which every thread keeps whether it waits or not).
// The wait is bounded; a copy that never lands is counted (the host turns the
// count into an error) and raises the CTA's abort flag: the caller stops
// updating and staging after the next barrier, and the kernel waits for the
// copies in flight once more before it exits (drain_copies).
// Returns whether this thread's wait saw the copy land.
__device__ __forceinline__ bool wait_staged(unsigned long long *bar, uint32_t phases, int b, unsigned &timeouts,
                                            int &abort)
{
    const bool ok = wait_parity_bounded(bar, (phases >> b) & 1u);
    if (!ok) {
        timeouts++;
        abort = 1;
    }
    return ok;
}

// Two FP32 values in one 64-bit register pair: the packed FP32 instructions
// (fma / mul .f32x2) do two lanes' worth of rounding-identical arithmetic per
// issue slot.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// VEC consecutive detector rows of one sinogram entry, as packed pairs.
template <int VEC>
struct Rows {
    f32x2 p[VEC / 2];
};
// e and w of one entry, loaded where i < n (else they keep what they hold): one
// predicate and two predicated loads, where an `if` compiles to a branch. e changes
// under the sweep (other CTAs' reductions land in L2), so it is read from there;
// w is constant.
__device__ __forceinline__ void load_entry(Rows<4> &e, Rows<4> &w, const float *pe, const float *pw, int i, int n)
{
    asm volatile(
        "{\n\t.reg .pred P;\n\tsetp.lt.s32 P, %6, %7;\n\t@P ld.global.cg.v2.b64 {%0, %1}, [%4];\n\t"
        "@P ld.global.nc.v2.b64 {%2, %3}, [%5];\n\t}"
        : "+l"(e.p[0]), "+l"(e.p[1]), "+l"(w.p[0]), "+l"(w.p[1])
        : "l"(pe), "l"(pw), "r"(i), "r"(n)
        : "memory");
}
__device__ __forceinline__ void load_entry(Rows<2> &e, Rows<2> &w, const float *pe, const float *pw, int i, int n)
{
    asm volatile(
        "{\n\t.reg .pred P;\n\tsetp.lt.s32 P, %4, %5;\n\t@P ld.global.cg.b64 %0, [%2];\n\t"
        "@P ld.global.nc.b64 %1, [%3];\n\t}"
        : "+l"(e.p[0]), "+l"(w.p[0])
        : "l"(pe), "l"(pw), "r"(i), "r"(n)
        : "memory");
}

// The generalised-Huber data term (XT_VoxUpdate.c:68-82): entries with |e sqrt(w)| >= T
// weigh T delta sqrt(w) / |e| instead of w.
//
// z = e^2 w against T^2 tells which they are, except within rounding of T^2. It is
// compared as bits, so that one maximum stands for an entry's rows (NaN and negative
// weights lie above all). The linear weight is q = a w / sqrt(z), a = T delta, from the
// hardware's approximate 1 / sqrt and a Newton step on q^2 e^2 = a^2 w. Against FP64 over
// w of 1e-11 to 1e11 and |e sqrt(w)| of T to 1e6 T it is off by at most 2.55 2^-24 (rms
// 0.60 to 0.67), as square root and division are by 1.96 to 3.83 (0.60 to 1.31).
//
// What this saves is code more than arithmetic. With both square roots and divisions
// inline at each of a batch's 16 pairs an iteration of 256 x 256 x 32 voxels in 8 frames
// (all entries linear at first, few at the end) took 35.7 to 28.0 ms; with the short form
// and them inline where it does not hold 36.6 to 30.6; without them 19.4 to 18.3; as a
// function of its own over the few pairs in question 21.3 to 18.5.
__device__ __forceinline__ unsigned top_bits(f32x2 v) { return max((unsigned)v, (unsigned)(v >> 32)); }

// the weights of the pairs `which` (bits), by square root and division
__device__ __noinline__ void huber_exact(const f32x2 *e, f32x2 *w, unsigned which, float T, float delta)
{
    auto weight = [=](float e_, float w_) {
        const float s = sqrtf(w_);
        return fabsf(e_ * s) < T ? w_ : T * delta * s / fmaxf(fabsf(e_), kMinNormal);  // T = 0: no weight, also at e = 0
    };
#pragma unroll 1
    for (; which; which &= which - 1) {
        const int k = __ffs(which) - 1;
        float e0, e1, w0, w1;
        unpack2(e[k], e0, e1);
        unpack2(w[k], w0, w1);
        w[k] = pack2(weight(e0, w0), weight(e1, w1));
    }
}

// the weights of a pair; sure: whether the short forms hold for both (else w comes back)
__device__ __forceinline__ f32x2 huber_pair(f32x2 e, f32x2 w, const IcdConst &K, bool &sure)
{
    const f32x2 z = mul2(mul2(e, e), w);
    float z0, z1, w0, w1, r0, r1, q0, q1;
    unpack2(z, z0, z1);
    unpack2(w, w0, w1);
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r0) : "f"(z0));
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r1) : "f"(z1));
    const f32x2 r = pack2(r0, r1);
    const f32x2 q = mul2(mul2(pack2(K.huber_a, K.huber_a), w), r), p = mul2(q, e);
    const f32x2 d = fma2(mul2(p, pack2(-1.0f, -1.0f)), p, mul2(pack2(K.huber_a2, K.huber_a2), w));  // a^2 w - q^2 e^2
    unpack2(fma2(d, mul2(r, pack2(K.huber_ha, K.huber_ha)), q), q0, q1);
    const bool quad0 = z0 < K.huber_T2 && w0 >= 0.0f, quad1 = z1 < K.huber_T2 && w1 >= 0.0f;
    // surely linear: T2hi <= z < kHuberMaxZ, kHuberMinW <= w < kHuberMaxW
    const unsigned z_lo = __float_as_uint(K.huber_T2hi), w_lo = __float_as_uint(kHuberMinW);
    auto lin = [&](float z_, float w_) {
        return __float_as_uint(z_) - z_lo < __float_as_uint(kHuberMaxZ) - z_lo &&
               __float_as_uint(w_) - w_lo < __float_as_uint(kHuberMaxW) - w_lo;
    };
    sure = (quad0 || lin(z0, w0)) && (quad1 || lin(z1, w1));
    return sure ? pack2(quad0 ? w0 : q0, quad1 ? w1 : q1) : w;
}

template <int VEC, int kBatch>
__device__ __forceinline__ void huber_weights(const Rows<VEC> (&e)[kBatch], Rows<VEC> (&w)[kBatch], const IcdConst &K)
{
    constexpr int P = VEC / 2;  // pairs an entry
    const unsigned limit = __float_as_uint(K.huber_T2);
    unsigned unsure = 0;
#pragma unroll
    for (int u = 0; u < kBatch; u++) {
        unsigned top = 0;
#pragma unroll
        for (int i = 0; i < P; i++) top = max(top, top_bits(mul2(mul2(e[u].p[i], e[u].p[i]), w[u].p[i])));
        if (top >= limit)
#pragma unroll
            for (int i = 0; i < P; i++) {
                bool sure;
                w[u].p[i] = huber_pair(e[u].p[i], w[u].p[i], K, sure);
                unsure |= sure ? 0u : 1u << (u * P + i);
            }
    }
    if (!unsure) return;
    f32x2 et[kBatch * P], wt[kBatch * P];
#pragma unroll
    for (int k = 0; k < kBatch * P; k++) et[k] = e[k / P].p[k % P], wt[k] = w[k / P].p[k % P];
    huber_exact(et, wt, unsure, K.huber_T, K.huber_delta);
#pragma unroll
    for (int k = 0; k < kBatch * P; k++) w[k / P].p[k % P] = wt[k];
}

// Vector reduction into global memory (red.global.add.v{2,4}.f32, sm_90+) where
// i < n: one predicated instruction (an `if` compiles to a branch).
__device__ __forceinline__ void red_add(float *p, const Rows<4> &d, int i, int n)
{
    float a, b, c, e;
    unpack2(d.p[0], a, b);
    unpack2(d.p[1], c, e);
    asm volatile(
        "{\n\t.reg .pred P;\n\tsetp.lt.s32 P, %5, %6;\n\t@P red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(p),
        "f"(a), "f"(b), "f"(c), "f"(e), "r"(i), "r"(n)
        : "memory");
}
__device__ __forceinline__ void red_add(float *p, const Rows<2> &d, int i, int n)
{
    float a, b;
    unpack2(d.p[0], a, b);
    asm volatile("{\n\t.reg .pred P;\n\tsetp.lt.s32 P, %3, %4;\n\t@P red.global.add.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p),
                 "f"(a), "f"(b), "r"(i), "r"(n)
                 : "memory");
}

struct IcdSmem {
    unsigned long long stage_bar[2];  // completion of the two record buffers' bulk copies
    float2 nd[kMaxWarps][32];         // per warp and slice: the prior's (num, den)
    float2 th[kMaxWarps][32];         // per warp and detector row: (theta1, theta2)
    unsigned pos[kMaxWarps];          // per warp: slices with a positive neighbour, as bits
    __align__(16) float dx[32];       // per detector row of the chunk: the change of its slice
    int2 order[kMaxSvCols];           // columns to visit: (index in the image, tile cell << 10 | sources inside the object)
    int ncols, item;
    int abort;              // a record copy did not land in time: stop updating
    unsigned issued[2];     // copies started into each buffer
};

struct IcdCount {
    unsigned long long upd, skip;
    float sum_dx, sum_x;
    unsigned timeouts;     // record copies that did not land in time
    uint32_t phases;       // parity of the next wait on each record buffer
};

// Warp 0 adds the CTA's counters to the problem's statistics and clears them.
__device__ __forceinline__ void flush_counts(IcdCount &cnt, IcdStats *stats)
{
    if ((threadIdx.x >> 5) == 0) {
        for (int off = 16; off > 0; off >>= 1) {
            cnt.upd += __shfl_xor_sync(0xffffffffu, cnt.upd, off);
            cnt.skip += __shfl_xor_sync(0xffffffffu, cnt.skip, off);
            cnt.sum_dx += __shfl_xor_sync(0xffffffffu, cnt.sum_dx, off);
            cnt.sum_x += __shfl_xor_sync(0xffffffffu, cnt.sum_x, off);
        }
        if ((threadIdx.x & 31) == 0 && (cnt.upd || cnt.skip)) {
            atomicAdd(&stats->updates, cnt.upd);
            atomicAdd(&stats->skipped, cnt.skip);
            atomicAdd(&stats->sum_abs_dx, (double)cnt.sum_dx);
            atomicAdd(&stats->sum_abs_x, (double)cnt.sum_x);
        }
    }
    if (cnt.timeouts && (threadIdx.x & 31) == 0) atomicAdd(&stats->stage_timeouts, cnt.timeouts);
    const uint32_t phases = cnt.phases;
    cnt = IcdCount{};
    cnt.phases = phases;
}

// Entry lists. A column's A records (header + values) are unpacked once into a
// list per view group of (sinogram offset, -a) pairs, a = A value x delta_t: the
// theta and apply passes then run over exactly the entries there are (2.27 a view
// at voxel scale 1, of the 3 slots of a record) without decoding or branching.
// A group's list: slot 0 holds its count and the largest count of the warp's
// groups, slots 1.. the entries, filled up with entries of weight zero to the
// multiple (at least one) of the batch that covers that largest count. `cap` slots a group, odd,
// so that the groups of a warp read different banks.
__host__ __device__ inline int icd_lanes_per_row(int N_t, int vec)  // lanes over a full chunk's rows, a power of two
{
    const int lpr = (N_t < 32 ? N_t : 32) / vec;
    int p = 1;
    while (p < lpr) p <<= 1;
    return p;
}
__host__ __device__ inline int icd_list_cap(int views_per_group, int kmax, int batch)
{
    return (1 + (views_per_group * kmax + batch - 1) / batch * batch) | 1;
}

// one entry, where i < n
__device__ __forceinline__ void put_entry(uint2 *p, unsigned off, float na, int i, int n)
{
    asm volatile("{\n\t.reg .pred P;\n\tsetp.lt.s32 P, %3, %4;\n\t@P st.shared.v2.b32 [%0], {%1, %2};\n\t}" ::"r"(
                     (unsigned)__cvta_generic_to_shared(p)),
                 "r"(off), "r"(__float_as_uint(na)), "r"(i), "r"(n)
                 : "memory");
}

// Unpack the records of view group `group` (views group, group + gstride, ...
// from v_begin below v_end) into `list`; called by all lanes of a warp, lane tq of
// the group's lprp lanes taking every lprp-th of its views.
template <int kBatch>
__device__ __forceinline__ void unpack_records(const uint32_t *rec, int RW, int NT, float dt, uint2 *list, int group,
                                               int gstride, int v_begin, int v_end, int tq, int lprp)
{
    int total = 0;
    for (int base = v_begin; base < v_end; base += gstride * lprp) {  // uniform over the CTA
        const int v = base + group + tq * gstride;
        const uint32_t *r = rec + (size_t)v * RW;
        uint4 head = make_uint4(0u, 0u, 0u, 0u);  // header and the first three values
        if (v < v_end) head = *reinterpret_cast<const uint4 *>(r);
        const int n = (int)(head.x >> 24);
        int incl = n;
        for (int o = 1; o < lprp; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o, lprp);
            if (tq >= o) incl += up;
        }
        uint2 *dst = list + 1 + total + incl - n;
        // sinogram rows stay below 2^24 and N_t rows each: 32-bit offsets
        const unsigned off = (head.x & 0xFFFFFFu) * (unsigned)NT;
        put_entry(dst, off, -(__uint_as_float(head.y) * dt), 0, n);
        put_entry(dst + 1, off + (unsigned)NT, -(__uint_as_float(head.z) * dt), 1, n);
        put_entry(dst + 2, off + 2u * (unsigned)NT, -(__uint_as_float(head.w) * dt), 2, n);
        for (int q = 3; q < n; q++)
            dst[q] = make_uint2(off + (unsigned)(q * NT), __float_as_uint(-(__uint_as_float(r[1 + q]) * dt)));
        total += __shfl_sync(0xffffffffu, incl, lprp - 1, lprp);
    }
    const int most = __reduce_max_sync(0xffffffffu, total);
    const int padded = max(1, (most + kBatch - 1) / kBatch) * kBatch;
    for (int i = total + tq; i < padded; i += lprp) list[1 + i] = make_uint2(0u, 0u);
    if (tq == 0) list[0] = make_uint2((unsigned)total, (unsigned)most);
}

// The in-plane and temporal neighbours ("sources") of a voxel column: s = 0..7
// the 3 x 3 neighbourhood in row-major order without its centre, 8 and 9 the
// same column in frames f - 1 and f + 1.
__device__ __forceinline__ void source_step(int s, int &dy, int &dx)
{
    const int o = s < 4 ? s : s + 1;
    dy = o / 3 - 1;
    dx = o - 3 * (dy + 1) - 1;
}

// sources of column (j, k) of frame f that lie inside the object, as bits
__device__ __forceinline__ int sources_inside(int j, int k, int f, int NX, int NY, int NT)
{
    int m = 0x3FF;
    if (j == 0) m &= ~0x007;
    if (j == NY - 1) m &= ~0x0E0;
    if (k == 0) m &= ~0x029;
    if (k == NX - 1) m &= ~0x094;
    if (f == 0) m &= ~0x100;
    if (f == NT - 1) m &= ~0x200;
    return m;
}

// r = h mod d for 1 <= d <= 2^16, in 32-bit steps
__device__ __forceinline__ unsigned mod_small(uint64_t h, unsigned d)
{
    const unsigned hi = (unsigned)(h >> 32), lo = (unsigned)h;
    return ((hi % d) * ((0xFFFFFFFFu % d + 1u) % d) + lo % d) % d;
}

// Update the voxel columns of super-voxel (sx, sy) of frame f; the whole CTA
// cooperates (see the file comment for the passes of a column).
// VEC: consecutive detector rows one lane owns (4 when N_t % 4 == 0, else 2);
// kStaged: a column's records arrive in shared memory by a TMA bulk copy (srec:
// two buffers) and are unpacked into entry lists while the column before it is
// solved; else the lists are unpacked from global memory, in blocks of views;
// kTile: the neighbours' values are read from the tile in shared memory
// (stage_tile), else from x;
// kHuber: 0 the quadratic data term, 1 the generalised Huber one
// (XT_VoxUpdate.c:68-82);
// kBatch: entries of a lane in flight together;
// kAnyZ: slices' rows need not divide a chunk of 32 (below).
//
// A view's entries are read (theta) and reduced into (apply) by the same lane
// for every column of the SV, so no barrier is needed between one column's
// apply pass and the next one's theta loads.
template <int VEC, bool kStaged, bool kTile, int kHuber, int kBatch, bool kAnyZ>
__device__ __forceinline__ void icd_update_sv(const Geom &g, const IcdLaunch &L, const IcdConst &K,
                                              const uint32_t *__restrict__ table,
                                              const int32_t *__restrict__ view_first,
                                              const uint8_t *__restrict__ mask, float *__restrict__ x,
                                              float *__restrict__ err, const float *__restrict__ wgt,
                                              float *__restrict__ mag, int f, int sx, int sy, IcdSmem &S,
                                              IcdCount &cnt, uint32_t *dyn)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const int NX = g.N_x, NY = g.N_y, NZ = g.N_z, NT = g.N_t, MZ = g.z_overlap;
    const int nxy = NX * NY;
    const int RW = g.rec_words;
    uint32_t *srec = dyn;
    uint2 *lists = reinterpret_cast<uint2 *>(dyn + (kStaged ? 2 * L.stage_words : 0));
    float *tile = reinterpret_cast<float *>(dyn + (kStaged ? 2 * L.stage_words : 0) + L.list_words) + 4;
    // A voxel column is updated in chunks of at most 32 detector rows (32 / MZ
    // voxel slices, one per lane of warp 0); chunk k covers rows [32k, 32k + 32)
    // and slices [k CZ, k CZ + CZ). Columns of up to 32 rows are one chunk.
    // kAnyZ (taller columns whose slices' rows, MZ, do not divide 32): a chunk is the
    // rows of its CZ slices (of one slice where MZ > 32), from wherever these begin.
    // Lanes hold two aligned rows (VEC 2), so the chunk is gone through in blocks of 32
    // rows from the aligned row at or before its first one; rows outside it count as
    // zero. MZ <= 31 gives one block (CZ MZ <= 31 and at most one row before them).
    static_assert(!kAnyZ || (VEC == 2 && !kStaged && !kTile), "any z scale: two rows a lane, lists from global memory");
    const int CT = NT < 32 ? NT : 32, CZ = kAnyZ ? max(1, 32 / MZ) : CT / MZ;
    const int n_chunks = kAnyZ ? (NZ + CZ - 1) / CZ : (NT + 31) / 32;

    // lane -> (view group, run of VEC detector rows) for the theta / apply passes
    const int lprp = icd_lanes_per_row(NT, VEC);
    const int G = 32 / lprp;  // view groups per warp
    const int grp = lane / lprp, tq = lane % lprp;
    const int t0 = tq * VEC;  // first detector row of this lane within the chunk
    const int gstride = W * G;
    // lane -> (neighbour source, slice) for the neighbourhood pass: a short
    // column leaves room for several sources side by side in a warp. The last
    // warps take the first in-plane sources (warp 0 has the solve to do), warps
    // from the second on the temporal ones.
    int zp = 1;
    while (zp < CZ) zp <<= 1;
    const int nsub = 32 / zp, sub = lane / zp, zlane = lane % zp;
    const int sfirst = (W - 1 - warp) * nsub, sstride = W * nsub;
    const int ts = (warp - (W >= 4 ? 1 : 0)) * nsub + sub;  // temporal source 8 + ts
    const int sv = L.sv, TW = sv + 2;  // the tile: the SV's columns and their in-plane neighbours
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const int iter = L.iter_dev ? *L.iter_dev : L.iter;  // 1-based iteration number
    const bool no_skip = !L.zero_skipping || iter <= 1;
    // entry lists: one per view group; two sets when staged (the current
    // column's and the next one's). Unstaged, the lists hold blocks of
    // L.block_views views.
    const int cap = L.list_cap, set_slots = gstride * cap;
    const uint32_t *rec_frame = table + (size_t)fv0 * nxy * RW;

    // ---- the SV's columns inside the reconstruction circle, shuffled ----------
    if (warp == 0) {
        const int ncand = sv * sv;
        int n = 0;
        for (int base = 0; base < ncand; base += 32) {
            const int i = base + lane;
            int ok = 0, c = 0, cell = 0;
            if (i < ncand) {
                const int j = sy * sv + i / sv, k = sx * sv + i % sv;
                if (j < NY && k < NX) {
                    c = j * NX + k;
                    cell = ((i / sv + 1) * TW + i % sv + 1) << 10 | sources_inside(j, k, f, NX, NY, g.N_time);
                    ok = mask[c] && (!L.sel || L.sel[(size_t)f * nxy + c]);
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) S.order[n + __popc(m & ((1u << lane) - 1))] = make_int2(c, cell);
            n += __popc(m);
        }
        __syncwarp();
        if (lane == 0) {
            uint64_t h = mix64(L.seed ^ mix64(((uint64_t)iter << 40) ^ ((uint64_t)f << 20) ^
                                             (uint64_t)(sy * L.n_sv_x + sx)));
            for (int i = n - 1; i > 0; i--) {  // Fisher-Yates
                h = mix64(h);
                const int r = (int)mod_small(h, (unsigned)(i + 1));
                const int2 t = S.order[i];
                S.order[i] = S.order[r];
                S.order[r] = t;
            }
            S.ncols = n;
        }
    }
    __syncthreads();
    const int ncols = S.ncols;
    if (ncols == 0) return;
    const bool starter = (int)threadIdx.x == 32 * (W - 1);  // starts the copies (not in warp 0, which solves)
    const bool tile_copy = kTile && NZ % 4 == 0;
    if (tile_copy) {
        // the tile's rows are contiguous in x: one bulk copy each, on the first
        // record buffer's mbarrier
        if (warp == W - 1) stage_tile(tile, x, g, f, sx, sy, sv, nv * RW * 4, &S.stage_bar[0]);
    } else if (kTile) {
        const int cells = 3 * TW * TW;
        for (int i = threadIdx.x; i < cells * NZ; i += blockDim.x) {
            const int cell = i / NZ, z = i - cell * NZ;
            const int p = cell / (TW * TW), r = cell - p * TW * TW;
            const int ff = p == 0 ? f : p == 1 ? f - 1 : f + 1, j = sy * sv - 1 + r / TW, k = sx * sv - 1 + r % TW;
            if (ff >= 0 && ff < g.N_time && j >= 0 && j < NY && k >= 0 && k < NX &&
                (p == 0 || (r / TW >= 1 && r / TW <= sv && r % TW >= 1 && r % TW <= sv)))
                tile[i] = x[((size_t)ff * nxy + (size_t)(j * NX + k)) * NZ + z];
        }
    }
    // copy column ci's records into buffer ci mod 2
    auto stage = [&](int ci) {
        if (starter && ci < ncols) {
            unsigned long long *bar = &S.stage_bar[ci & 1];
            if (ci > 0 || !tile_copy) expect_bytes(bar, nv * RW * 4);
            S.issued[ci & 1]++;
            if (nv) bulk_copy(srec + (ci & 1) * L.stage_words, rec_frame + (size_t)S.order[ci].x * nv * RW, 4u * (unsigned)(nv * RW), bar);
        }
    };
    if (kStaged) stage(0);

    // filter coefficients (with the 1 / sigma^q) of the neighbours at distance 1,
    // sqrt 2 and sqrt 3
    const float f1 = K.sf[9 + 1] * K.issq, f2 = K.sf[9] * K.issq, f3 = K.sf[0] * K.issq;

    int2 next = make_int2(0, 0);
    // ci = -1 only unpacks the first column's records
    for (int ci = kStaged ? -1 : 0; ci < ncols; ci++) {
        const int2 col = kStaged ? next : S.order[ci];
        if (kStaged && ci + 1 < ncols) next = S.order[ci + 1];
        const int c = col.x, inside = col.y & 0x3FF;
        const size_t col_off = ((size_t)f * nxy + c) * NZ;
        float *cb = kTile ? tile + (col.y >> 10) * NZ : x + col_off;  // the column's values
        const uint2 *ent = lists + (kStaged ? (ci & 1) * set_slots : 0) + (warp * G + grp) * cap;

        for (int ch = 0; ch < n_chunks; ch++) {
            const int z0 = ch * CZ;                                  // first slice of the chunk
            const int cz = NZ - z0 < CZ ? NZ - z0 : CZ;              // slices in the chunk
            const int first_row = kAnyZ ? z0 * MZ : ch * 32, end_row = first_row + cz * MZ;  // the chunk's rows
            const int rbase = kAnyZ ? first_row & ~(VEC - 1) : first_row;  // first row of its first block
            int rb = rbase;                                                // of the current block
            bool row_ok = kAnyZ ? rb + t0 < end_row : tq < cz * MZ / VEC;
            unsigned rows0 = (unsigned)(rb + t0);  // this lane's rows within an entry
            // (kAnyZ) go on to the chunk's next block of rows
            auto next_rows = [&]() {
                rb += 32;
                row_ok = rb + t0 < end_row;
                rows0 = (unsigned)(rb + t0);
                return rb < end_row;
            };
            bool active = ci >= 0;
            float V = 0.0f;
            int vb = 0;
            // (unstaged: the lists hold a block of the column's views at a time)
            auto next_block = [&]() {
                __syncwarp();
                unpack_records<kBatch>(rec_frame + (size_t)c * nv * RW, RW, NT, K.dt, lists + (warp * G + grp) * cap,
                                       warp * G + grp, gstride, vb, min(vb + L.block_views, nv), tq, lprp);
                __syncwarp();
            };
            if (ci >= 0) {
                const bool zl = zlane < cz;
                const int z = z0 + zlane;  // this lane's slice
                const float v0 = kTile || zl ? cb[z] : 0.0f;
                V = zl ? v0 : 0.0f;
                const bool sure = no_skip || __any_sync(0xffffffffu, zl && V != 0.0f);
                // theta's first batch of entries is in flight during the
                // neighbourhood pass (e and w keep the last values loaded: an entry
                // that is not there has weight zero)
                Rows<VEC> e[kBatch], w[kBatch];
                float na[kBatch];
                f32x2 t1[VEC / 2], t2[VEC / 2];
#pragma unroll
                for (int u = 0; u < kBatch; u++) e[u] = w[u] = Rows<VEC>{};
#pragma unroll
                for (int i = 0; i < VEC / 2; i++) t1[i] = t2[i] = 0ull;
                if (!kStaged) next_block();
                int n_ent = row_ok ? (int)ent[0].x : 0, n_warp = (int)ent[0].y, i0 = 0;
                bool first = true;
                for (;;) {  // once; kAnyZ: the chunk's blocks of rows
                    for (;;) {
                        // entries i0 .. i0 + kBatch - 1: all loads in flight together
#pragma unroll
                        for (int u = 0; u < kBatch; u++) {
                            const uint2 en = ent[1 + i0 + u];
                            const unsigned off = en.x + rows0;
                            na[u] = __uint_as_float(en.y);
                            load_entry(e[u], w[u], err + off, wgt + off, i0 + u, n_ent);
                        }
                        // ---- 1. neighbourhood, while the first batch arrives (sources
                        //         split over warps and lane groups) ------------------------
                        if (first) {
                            first = false;
                            float num = 0.0f, den = 0.0f, top = 0.0f;  // top: the largest neighbour, or 0
                            const bool zm = z > 0, zn = z + 1 < NZ;
                            for (int s0 = sfirst; s0 < 8; s0 += sstride) {  // in-plane; uniform over the warp
                                const int s = min(s0 + sub, 7);
                                int dy, dx;
                                source_step(s, dy, dx);
                                const bool ok = zl && s0 + sub < 8 && ((inside >> s) & 1), side = dy == 0 || dx == 0;
                                const float *src = cb + (ptrdiff_t)((dy * (kTile ? TW : NX) + dx) * NZ);
                                float n[3], d[3], fl[3], cf[3];
                                // (in the tile every address read exists: values outside the
                                // object are dropped after the load, without a branch)
                                const float nm = kTile || (ok && zm) ? src[z - 1] : 0.0f;
                                const float n0 = kTile || ok ? src[z] : 0.0f;
                                const float np = kTile || (ok && zn) ? src[z + 1] : 0.0f;
                                n[0] = ok && zm ? nm : 0.0f;
                                n[1] = ok ? n0 : 0.0f;
                                n[2] = ok && zn ? np : 0.0f;
                                const float fo = side ? f2 : f3;
                                fl[0] = ok && zm ? fo : 0.0f;
                                fl[1] = ok ? (side ? f1 : f2) : 0.0f;
                                fl[2] = ok && zn ? fo : 0.0f;
#pragma unroll
                                for (int i = 0; i < 3; i++) d[i] = V - n[i];
                                qg_coef(d, fl, K.q, K.qmp, K.issqp, K.cs, K.qocs, cf);
#pragma unroll
                                for (int i = 0; i < 3; i++) {
                                    num += cf[i] * n[i];
                                    den += cf[i];
                                    top = fmaxf(top, n[i]);
                                }
                            }
                            // temporal (the same source for every lane of a lane group)
                            for (int t0_ = ts - sub; t0_ < 2 && t0_ >= 0; t0_ += sstride) {
                                const int t = min(t0_ + sub, 1);
                                const bool ok = zl && t0_ + sub < 2 && ((inside >> (8 + t)) & 1);
                                const float *src = kTile ? cb + (t + 1) * TW * TW * NZ
                                                         : cb + (t == 0 ? -(ptrdiff_t)nxy : (ptrdiff_t)nxy) * NZ;
                                const float n0 = kTile || ok ? src[z] : 0.0f;
                                const float n[1] = {ok ? n0 : 0.0f}, d[1] = {V - n[0]}, fl[1] = {ok ? K.tf * K.istq : 0.0f};
                                float cf[1];
                                qg_coef(d, fl, K.q, K.qmp, K.istqp, K.ct, K.qoct, cf);
                                num += cf[0] * n[0];
                                den += cf[0];
                                top = fmaxf(top, n[0]);
                            }
                            unsigned pw = __ballot_sync(0xffffffffu, top > 0.0f);
                            for (int off = zp; off < 32; off <<= 1) {
                                num += __shfl_xor_sync(0xffffffffu, num, off);
                                den += __shfl_xor_sync(0xffffffffu, den, off);
                                pw |= pw >> off;
                            }
                            if (sub == 0) S.nd[warp][zlane] = make_float2(num, den);
                            if (lane == 0) S.pos[warp] = pw & (0xffffffffu >> (32 - zp));
                            // a column that may be inactive (all of it zero) needs the
                            // neighbours' verdict first (uniform: every warp read the column)
                            if (!sure) {
                                __syncthreads();
                                unsigned any = 0;
                                for (int q = 0; q < W; q++) any |= S.pos[q];
                                active = any != 0;
                                if (!active) break;
                            }
                        }
                        // ---- 2. theta1 = -sum a w e, theta2 = sum a^2 w over the column's
                        //         entries (XT_VoxUpdate.c:56-85) ---------------------------
                        if (kHuber) huber_weights(e, w, K);
#pragma unroll
                        for (int u = 0; u < kBatch; u++) {
                            const f32x2 a = pack2(na[u], na[u]);
#pragma unroll
                            for (int i = 0; i < VEC / 2; i++) {
                                const f32x2 aw = mul2(a, w[u].p[i]);  // -a w
                                t2[i] = fma2(a, aw, t2[i]);
                                t1[i] = fma2(e[u].p[i], aw, t1[i]);
                            }
                        }
                        i0 += kBatch;
                        if (i0 >= n_warp) {  // uniform over the warp
                            vb += L.block_views;
                            if (kStaged || vb >= nv) break;
                            next_block();
                            n_ent = row_ok ? (int)ent[0].x : 0;
                            n_warp = (int)ent[0].y;
                            i0 = 0;
                        }
                    }
                    if (active) {
                        // sum over the warp's view groups: two groups share out their rows
                        // until a lane holds one row, then add it up over the rest
                        float a[VEC], b[VEC];
#pragma unroll
                        for (int i = 0; i < VEC / 2; i++) {
                            unpack2(t1[i], a[2 * i], a[2 * i + 1]);
                            unpack2(t2[i], b[2 * i], b[2 * i + 1]);
                        }
                        int row = t0, off = lprp;
#pragma unroll
                        for (int n = VEC / 2; n >= 1; n /= 2) {
                            const bool up = (lane & off) != 0;
#pragma unroll
                            for (int i = 0; i < n; i++) {
                                const float sa = up ? a[i] : a[n + i], sb = up ? b[i] : b[n + i];
                                a[i] = (up ? a[n + i] : a[i]) + __shfl_xor_sync(0xffffffffu, sa, off);
                                b[i] = (up ? b[n + i] : b[i]) + __shfl_xor_sync(0xffffffffu, sb, off);
                            }
                            row += up ? n : 0;
                            off <<= 1;
                        }
                        const bool writes = lane < off && row_ok;
                        for (; off < 32; off <<= 1) {
                            a[0] += __shfl_xor_sync(0xffffffffu, a[0], off);
                            b[0] += __shfl_xor_sync(0xffffffffu, b[0], off);
                        }
                        if (!kAnyZ) {
                            if (writes) S.th[warp][row] = make_float2(a[0], b[0]);
                        } else if (writes) {
                            // rows outside the chunk are zero; a slice of several blocks adds
                            // them up (the same lane holds a row of every block)
                            const bool in = rb + row >= first_row && rb + row < end_row;
                            const float2 sum = rb == rbase ? make_float2(0.0f, 0.0f) : S.th[warp][row];
                            S.th[warp][row] = make_float2(sum.x + (in ? a[0] : 0.0f), sum.y + (in ? b[0] : 0.0f));
                        }
                    }
                    if (!kAnyZ || !active || !next_rows()) break;
                    vb = 0;
                    next_block();
                    n_ent = row_ok ? (int)ent[0].x : 0, n_warp = (int)ent[0].y, i0 = 0;
#pragma unroll
                    for (int i = 0; i < VEC / 2; i++) t1[i] = t2[i] = 0ull;
                }
            }
            __syncthreads();

            // while warp 0 solves, the other warps unpack the next column's records
            // (warp 1 also warp 0's share), and the copy of the column after it
            // starts, into the buffer that the current column's were unpacked from
            if (kStaged && (ch == n_chunks - 1 || ci < 0) && ci + 1 < ncols) {
                const int b = (ci + 1) & 1;
                stage(ci + 2);
                if ((warp > 0 || W == 1 || ci < 0) &&
                    wait_staged(&S.stage_bar[b], cnt.phases, b, cnt.timeouts, S.abort) && (warp > 0 || W == 1)) {
                    for (int q = warp; q >= 0; q = q == 1 ? 0 : -1)
                        unpack_records<kBatch>(srec + b * L.stage_words, RW, NT, K.dt,
                                               lists + b * set_slots + (q * G + grp) * cap, q * G + grp, gstride, 0, nv, tq,
                                               lprp);
                }
                cnt.phases ^= 1u << b;
            }

            // ---- 3. zero-skipping and solve (warp 0, lane = slice of the chunk) --------
            if (warp == 0 && ci >= 0) {
                const bool sl = lane < cz;
                if (!active) {
                    if (sl) cnt.skip++;
                    if (lane == 0 && ch == 0) mag[(size_t)f * nxy + c] = 0.0f;
                } else {
                    const int sz = z0 + lane;
                    const bool has_m = sl && sz >= 1, has_p = sl && sz + 1 < NZ;
                    const float fv[2] = {has_m ? f1 : 0.0f, has_p ? f1 : 0.0f};
                    // in-column z - 1 / z + 1: the chunk below is already updated
                    // (Gauss-Seidel over the chunks), the chunk above not yet
                    float vm = has_m ? cb[sz - 1] : 0.0f, vp = has_p ? cb[sz + 1] : 0.0f;
                    float numA = 0.0f, denA = 0.0f, th1 = 0.0f, th2 = 0.0f;
                    unsigned pw = 0;
#pragma unroll 4
                    for (int q = 0; q < W; q++) {
                        const float2 nd = S.nd[q][lane], th = S.th[q][lane];
                        numA += nd.x;
                        denA += nd.y;
                        th1 += th.x;
                        th2 += th.y;
                        pw |= S.pos[q];
                    }
                    const bool pos = ((pw >> lane) & 1u) || vm > 0.0f || vp > 0.0f;
                    const bool skip = !sl || (!no_skip && V == 0.0f && !pos);
                    if (MZ > 1) {  // a slice covers MZ detector rows
                        __syncwarp();
                        S.th[0][lane] = make_float2(th1, th2);
                        __syncwarp();
                        th1 = th2 = 0.0f;
                        if (!kAnyZ && sl) {
                            for (int r = 0; r < MZ; r++) {
                                const float2 th = S.th[0][lane * MZ + r];
                                th1 += th.x;
                                th2 += th.y;
                            }
                        } else if (sl) {  // the rows of the slice's block, or (one slice) of all blocks
                            const int r0 = CZ == 1 ? 0 : first_row - rbase + lane * MZ;
                            const int r1 = CZ == 1 ? min(32, end_row - rbase) : r0 + MZ;
                            for (int r = r0; r < r1; r++) {
                                const float2 th = S.th[0][r];
                                th1 += th.x;
                                th2 += th.y;
                            }
                        }
                    }
                    // even slices, then odd ones against the even ones' new values (the
                    // other lanes' results are dropped)
                    float cur = V;
#pragma unroll 1
                    for (int parity = 0; parity < 2; parity++) {
                        const float d[2] = {V - vm, V - vp};
                        float cv[2];
                        qg_coef(d, fv, K.q, K.qmp, K.issqp, K.cs, K.qocs, cv);
                        if (!skip && (sz & 1) == parity) {
                            const float num = (numA + cv[0] * vm) + cv[1] * vp;
                            const float den = (denA + cv[0]) + cv[1];
                            const float u = (num + th2 * V - th1) / (den + th2);
                            cur = V + K.alpha * (u - V);
                        }
                        const float um = __shfl_up_sync(0xffffffffu, cur, 1), up = __shfl_down_sync(0xffffffffu, cur, 1);
                        if (has_m && lane > 0) vm = um;  // across chunk edges: the values read above
                        if (has_p && lane < cz - 1) vp = up;
                    }
                    const float dx = skip ? 0.0f : cur - V;
                    S.dx[lane] = MZ == 1 || kAnyZ ? dx : __shfl_sync(0xffffffffu, dx, lane / MZ);  // kAnyZ: by slice
                    if (sl && !skip) {
                        x[col_off + sz] = cur;
                        if (kTile) cb[sz] = cur;
                        cnt.upd++;
                        cnt.sum_dx += fabsf(dx);
                        cnt.sum_x += fabsf(cur);
                    }
                    if (sl && skip) cnt.skip++;
                }
            }
            __syncthreads();
            // a late copy leaves the next column's records undefined: no further
            // update, no further copies (uniform: the flag was set before the barrier)
            if (S.abort) return;
            if (ci < 0) break;
            if (!active) continue;

            // ---- 4. apply e -= a dx ------------------------------------------------------
            {
                auto apply = [&](const Rows<VEC> &dxv) {
                    bool any = false;
#pragma unroll
                    for (int i = 0; i < VEC / 2; i++) any |= (dxv.p[i] & 0x7FFFFFFF7FFFFFFFull) != 0;
                    any = __any_sync(0xffffffffu, any);
                    if (!any) return;
                    for (vb = 0;;) {
                        if (!kStaged && L.block_views < nv) next_block();
                        const int n = row_ok ? (int)ent[0].x : 0, n_warp = (int)ent[0].y;
                        for (int i0 = 0; i0 < n_warp; i0 += 4) {  // uniform over the warp
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                const uint2 en = ent[1 + i0 + u];
                                const float na = __uint_as_float(en.y);
                                const f32x2 a = pack2(na, na);
                                Rows<VEC> d;
#pragma unroll
                                for (int q = 0; q < VEC / 2; q++) d.p[q] = mul2(a, dxv.p[q]);
                                red_add(err + (en.x + rows0), d, i0 + u, n);
                            }
                        }
                        vb += L.block_views;
                        if (kStaged || vb >= nv) break;
                    }
                };
                if constexpr (!kAnyZ) {
                    Rows<VEC> dxv{};
                    if (row_ok) dxv = *reinterpret_cast<const Rows<VEC> *>(&S.dx[t0]);
                    apply(dxv);
                } else {
                    auto dx_of = [&](int r) { return r >= first_row && r < end_row ? S.dx[(r - first_row) / MZ] : 0.0f; };
                    rb = rbase - 32;
                    while (next_rows()) apply(Rows<VEC>{{pack2(dx_of(rb + t0), dx_of(rb + t0 + 1))}});
                }
                // the column's update magnitude: the sum over its slices of |dx| (by
                // the last warp: warp 0's chain is the longest)
                if (warp == W - 1) {
                    float m = (kAnyZ ? lane < cz : lane < cz * MZ && lane % MZ == 0) ? fabsf(S.dx[lane]) : 0.0f;
                    for (int off = 16; off > 0; off >>= 1) m += __shfl_xor_sync(0xffffffffu, m, off);
                    if (lane == 0) {
                        float *mp = mag + (size_t)f * nxy + c;
                        *mp = ch == 0 ? m : *mp + m;
                    }
                }
            }
        }
    }
    // the next SV's tile is written by the copy engine over these generic writes
    if (kTile) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

}  // namespace

__device__ __forceinline__ void init_copies(IcdSmem &S)
{
    if (threadIdx.x == 0) {
        S.abort = 0;
        for (int b = 0; b < 2; b++) {
            S.issued[b] = 0;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&S.stage_bar[b]))
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// After an abort, copies may still write into this CTA's shared memory: give
// the last one of each buffer one more bounded wait before the CTA exits.
__device__ __forceinline__ void drain_copies(IcdSmem &S)
{
    if (S.abort && threadIdx.x == 0)
        for (int b = 0; b < 2; b++)
            if (S.issued[b]) wait_parity_bounded(&S.stage_bar[b], (S.issued[b] - 1) & 1u);
}

// One colour phase of one problem: persistent CTAs drain the phase's SV queue.
// 128 registers a thread: four CTAs of four warps on an SM, which is what the
// batch of loads in flight needs; at 72 registers (seven CTAs) the spills cost
// more than the occupancy gave (4-D workload, iteration with its NH passes: 16.1
// against 12.0 ms).
template <int VEC, bool kStaged, bool kTile, int kHuber, int kBatch, bool kAnyZ>
__global__ void __launch_bounds__(kMaxWarps * 32, 2) icd_phase_kernel(
    Geom g, IcdLaunch L, IcdConst K, const uint32_t *__restrict__ table, const int32_t *__restrict__ view_first,
    const uint8_t *__restrict__ mask, float *__restrict__ x, float *__restrict__ err, const float *__restrict__ wgt,
    float *__restrict__ mag, IcdStats *__restrict__ stats, unsigned int *__restrict__ queue)
{
    __shared__ IcdSmem S;
    extern __shared__ __align__(16) uint32_t s_dyn[];
    const int KC = L.colors_k;
    const int hx = (L.n_sv_x + KC - 1) / KC, slots = hx * ((L.n_sv_y + KC - 1) / KC);
    const int n_items = L.items ? *L.n_items : g.N_time * slots;
    IcdCount cnt{};
    init_copies(S);
    for (;;) {
        __syncthreads();  // S.item / S.order of the previous SV are no longer read
        if (S.abort) break;  // uniform: written before the barrier
        if (threadIdx.x == 0) S.item = (int)atomicAdd(queue, 1u);
        __syncthreads();
        const int item = S.item;
        if (item >= n_items) break;
        int f, sx, sy;
        if (L.items) {  // explicit work list (its SVs hold columns to update)
            const uint32_t code = L.items[item];
            f = (int)(code >> 22);
            sy = (int)((code >> 11) & 2047u);
            sx = (int)(code & 2047u);
        } else {
            f = item % g.N_time;  // frames fastest: concurrent SVs spread over the frames
            const int rem = (int)((long long)(item / g.N_time) * L.perm % slots);
            const int color = (L.phase + f) % (KC * KC);  // frame f +- 1 is never on the same colour
            sx = KC * (rem % hx) + color % KC;
            sy = KC * (rem / hx) + color / KC;
        }
        if (sx >= L.n_sv_x || sy >= L.n_sv_y) continue;  // uniform
        icd_update_sv<VEC, kStaged, kTile, kHuber, kBatch, kAnyZ>(g, L, K, table, view_first, mask, x, err, wgt, mag, f,
                                                                  sx, sy, S, cnt, s_dyn);
    }
    drain_copies(S);
    flush_counts(cnt, stats);
}

// Shared memory of a launch (the fields of L that describe it; returns whether
// records are staged). Records and two sets of entry lists are staged up to
// kMaxStageBytes; beyond (thousands of views in a frame) lists of kBlockBytes
// are unpacked from global memory where they are used. An SV's neighbourhood tile
// (three planes of (sv + 2)^2 columns) is kept up to kMaxTileBytes; beyond, the
// neighbours are read from x where they are used.
constexpr size_t kMaxStageBytes = 128 * 1024, kBlockBytes = 16 * 1024, kMaxTileBytes = 40 * 1024;

// What a sweep keeps in shared memory: a block of entry lists only; or two record
// buffers and the lists of two columns; or these and the SV's neighbourhood tile.
enum IcdMode { ICD_PLAIN, ICD_STAGED, ICD_STAGED_TILE };
static IcdMode icd_plan_shared(const Geom &g, IcdLaunch &L, int vec, int batch, IcdMode most = ICD_STAGED_TILE)
{
    const int gstride = L.warps * (32 / icd_lanes_per_row(g.N_t, vec));
    const int vpg = std::max(1, (g.max_views + gstride - 1) / gstride);
    L.stage_words = g.max_views * g.rec_words;
    L.list_cap = icd_list_cap(vpg, g.kmax, batch);
    L.block_views = vpg * gstride;
    size_t lists = (size_t)gstride * L.list_cap * sizeof(uint2);
    const size_t records = L.stage_words * sizeof(uint32_t);
    const size_t tile = 3 * (size_t)(L.sv + 2) * (L.sv + 2) * g.N_z * sizeof(float);
    IcdMode mode = ICD_PLAIN;
    if (L.stage_records && most >= ICD_STAGED && 2 * (records + lists) <= kMaxStageBytes) {
        mode = most == ICD_STAGED_TILE && tile <= kMaxTileBytes ? ICD_STAGED_TILE : ICD_STAGED;
        lists *= 2;
    } else if (lists > kBlockBytes) {
        int v = vpg;
        while (v > 1 && (size_t)gstride * icd_list_cap(v, g.kmax, batch) * sizeof(uint2) > kBlockBytes) v--;
        L.list_cap = icd_list_cap(v, g.kmax, batch);
        L.block_views = v * gstride;
        lists = (size_t)gstride * L.list_cap * sizeof(uint2);
    }
    L.list_words = (int)((lists + 15) / 16 * 4);
    L.shared_bytes = (mode != ICD_PLAIN ? 2 * (int)records : 0) + 4 * L.list_words + (mode == ICD_STAGED_TILE ? (int)tile + 64 : 0);
    return mode;
}

template <int VEC, bool kStaged, bool kTile, int kHuber, int kBatch, bool kAnyZ = false>
static void launch_mode(const Geom &g, const IcdLaunch &L, const IcdConst &K, const uint32_t *d_table,
                        const int32_t *d_view_first, const uint8_t *d_mask, float *d_x, float *d_err,
                        const float *d_w, float *d_mag, IcdStats *d_stats, unsigned int *d_queue, cudaStream_t st)
{
    const int threads = L.warps * 32;
    const size_t smem = (size_t)L.shared_bytes;
    const auto kernel = icd_phase_kernel<VEC, kStaged, kTile, kHuber, kBatch, kAnyZ>;
    // resident CTAs per SM, cached per (device, block size, shared memory) so a
    // launch being captured into a CUDA graph makes no occupancy query
    struct Occ {
        int dev, threads, sms, per_sm;
        size_t smem;
    };
    static std::mutex mu;
    static std::vector<Occ> cache;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lk(mu);
        bool hit = false;
        for (const Occ &o : cache)
            if (o.dev == dev && o.threads == threads && o.smem == smem) {
                sms = o.sms;
                per_sm = o.per_sm;
                hit = true;
                break;
            }
        if (!hit) {
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMaxStageBytes + kMaxTileBytes));
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
            cache.push_back({dev, threads, sms, per_sm, smem});
        }
    }
    const long long items = (long long)g.N_time * sv_slots(g.N_x, g.N_y, L.sv, L.colors_k);
    long long grid = (long long)sms * (per_sm > 0 ? per_sm : 1);
    if (grid > items) grid = items;
    if (L.max_ctas > 0 && grid > L.max_ctas) grid = L.max_ctas;
    kernel<<<(unsigned)grid, threads, smem, st>>>(g, L, K, d_table, d_view_first, d_mask, d_x, d_err, d_w, d_mag,
                                                  d_stats, d_queue);
}

template <int VEC, int kBatch>
static void launch_vec(const Geom &g, const IcdLaunch &L_, const IcdConst &K, const uint32_t *d_table,
                       const int32_t *d_view_first, const uint8_t *d_mask, float *d_x, float *d_err, const float *d_w,
                       float *d_mag, IcdStats *d_stats, unsigned int *d_queue, cudaStream_t st)
{
    IcdLaunch L = L_;
    const IcdMode mode = icd_plan_shared(g, L, VEC, kBatch);
#define MBIR_MODE(S, T)                                                                                       \
    (K.huber ? launch_mode<VEC, S, T, 1, kBatch> : launch_mode<VEC, S, T, 0, kBatch>)(                          \
        g, L, K, d_table, d_view_first, d_mask, d_x, d_err, d_w, d_mag, d_stats, d_queue, st)
    if (mode == ICD_STAGED_TILE) MBIR_MODE(true, true);
    else if (mode == ICD_STAGED) MBIR_MODE(true, false);
    else MBIR_MODE(false, false);
#undef MBIR_MODE
}

// Columns of more than 32 rows whose slices' rows do not divide 32 (z scales that are no
// power of two, or above 32): the lists come from global memory, two rows a lane.
static void launch_any_z(const Geom &g, const IcdLaunch &L_, const IcdConst &K, const uint32_t *d_table,
                         const int32_t *d_view_first, const uint8_t *d_mask, float *d_x, float *d_err, const float *d_w,
                         float *d_mag, IcdStats *d_stats, unsigned int *d_queue, cudaStream_t st)
{
    IcdLaunch L = L_;
    icd_plan_shared(g, L, 2, 8, ICD_PLAIN);
    (K.huber ? launch_mode<2, false, false, 1, 8, true> : launch_mode<2, false, false, 0, 8, true>)(
        g, L, K, d_table, d_view_first, d_mask, d_x, d_err, d_w, d_mag, d_stats, d_queue, st);
}

IcdConst make_icd_const(const Geom &g)
{
    IcdConst K;
    for (int i = 0; i < 27; i++) K.sf[i] = (float)g.spatial_filter[i];
    K.tf = (float)g.time_filter;
    K.q = (float)g.q;
    K.qmp = (float)(g.q - g.p);
    K.issq = (float)(1.0 / g.sigma_s_q);
    K.issqp = (float)(1.0 / g.sigma_s_q_p);
    K.istq = (float)(1.0 / g.sigma_t_q);
    K.istqp = (float)(1.0 / g.sigma_t_q_p);
    K.cs = (float)g.c_s;
    K.ct = (float)g.c_t;
    K.qocs = (float)(g.q / g.c_s);
    K.qoct = (float)(g.q / g.c_t);
    K.bs0 = (float)(g.q / (g.sigma_s_q * g.c_s));
    K.bt0 = (float)(g.q / (g.sigma_t_q * g.c_t));
    K.alpha = (float)g.alpha;
    K.dt = (float)g.delta_t;
    K.huber_T = (float)g.huber_T;
    K.huber_delta = (float)g.huber_delta;
    K.huber_T2 = (float)(g.huber_T * g.huber_T * (1.0 - 1e-5));
    K.huber_T2hi = (float)(g.huber_T * g.huber_T * (1.0 + 1e-5));
    const double a = g.huber_T * g.huber_delta;
    K.huber_a = (float)a;
    K.huber_a2 = (float)(a * a);
    K.huber_ha = (float)(0.5 / a);
    // beyond these the short form's products may leave FP32's range: no entry is then surely linear
    if (!(a > 1e-4 && a < 1e4 && g.huber_T > 1e-8 && K.huber_T2hi < kHuberMaxZ)) K.huber_T2hi = kHuberMaxZ;
    K.huber = g.huber;
    return K;
}

void launch_icd_phase(const Geom &g, const IcdLaunch &L, const uint32_t *d_table, const int32_t *d_view_first,
                      const uint8_t *d_mask, float *d_x, float *d_err, const float *d_w, float *d_mag,
                      IcdStats *d_stats, unsigned int *d_queue, cudaStream_t st)
{
    const IcdConst K = make_icd_const(g);
    if (g.N_t > 32 && 32 % g.z_overlap) {
        launch_any_z(g, L, K, d_table, d_view_first, d_mask, d_x, d_err, d_w, d_mag, d_stats, d_queue, st);
        return;
    }
    const bool v4 = g.N_t % 4 == 0;
    // entries in flight: 8, or 4 where no view group has more (one view each: a
    // batch is then mostly filling), or as the caller asks
    const int gstride = L.warps * (32 / icd_lanes_per_row(g.N_t, v4 ? 4 : 2));
    const int most = (g.max_views + gstride - 1) / gstride * g.kmax;
    const bool b8 = L.unroll > 0 ? L.unroll >= 2 : most > 4;
    const auto launch = v4 ? (b8 ? launch_vec<4, 8> : launch_vec<4, 4>) : (b8 ? launch_vec<2, 8> : launch_vec<2, 4>);
    launch(g, L, K, d_table, d_view_first, d_mask, d_x, d_err, d_w, d_mag, d_stats, d_queue, st);
}

}  // namespace mbirgpu
