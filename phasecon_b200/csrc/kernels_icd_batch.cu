// Batched super-voxel ICD: one colour phase of many independent problems in one
// persistent launch.
//
// The column update of this kernel reads records, e and w straight from global memory,
// without the one-problem sweep's staging, entry lists and tile (kernels_icd.cu). In a
// batch nearly all super-voxels of a phase are in flight at once, and which of their
// updates see each other's is part of the method: the lists' update in the same grid
// gave an iteration in 10.6 ms instead of 16.1 (12 problems of 64 x 64 x 8 to
// 256 x 256 x 32 voxels), but images that still move, 16 iterations from zero, were
// then further from this kernel's than four times what two runs of it differ by, at
// the rim of the reconstruction circle; staging with its tile (three CTAs on an SM)
// converged at half the pace.
#include "mbir_internal.h"

namespace mbirgpu {

namespace {

constexpr int kMaxWarps = 8;
constexpr int kMaxSvCols = 256;  // sv <= 16
constexpr float kMinNormal = 1.17549435e-38f;  // 2^-126

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
// t3 = c + t1. Takes isq = 1 / sq and isqp = 1 / sqp. The weight is
// evaluated ~28 times per voxel update, so it uses the hardware base-2
// logarithm / exponential (one logarithm for both powers) and reciprocal:
// FP32 arithmetic whose rounding the FP64 MAP cost, by which the method's
// result is measured, does not see. Differences below 2^-126 count as zero: the
// logarithm takes them for it.
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
__device__ __forceinline__ float qg_weight(float d, float q, float qmp, float isq, float isqp, float c, float b0)
{
    if (fabsf(d) < kMinNormal) return b0;
    const float l = lg2_hw(fabsf(d));
    const float t1 = ex2_hw(qmp * l) * isqp;
    const float rt3 = rcp_hw(c + t1);
    float r = (q - qmp * t1 * rt3) * rt3 * isq;
    if (q != 2.0f) r *= ex2_hw((q - 2.0f) * l);
    return r;
}

// A record: header and three values (a batch's problems have voxel scale 1).
__device__ __forceinline__ float rec_val(const uint4 &r, int q)
{
    return __uint_as_float(q == 0 ? r.y : q == 1 ? r.z : r.w);
}

template <int VEC>
struct VecF;
template <>
struct VecF<4> {
    using T = float4;
    __device__ static void get(const T &v, float *o) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
};
template <>
struct VecF<2> {
    using T = float2;
    __device__ static void get(const T &v, float *o) { o[0] = v.x; o[1] = v.y; }
};

// Vector reduction into global memory (red.global.add.v{2,4}.f32, sm_90+).
__device__ __forceinline__ void red_add(float *p, const float (&d)[4])
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(d[0]), "f"(d[1]), "f"(d[2]), "f"(d[3])
                 : "memory");
}
__device__ __forceinline__ void red_add(float *p, const float (&d)[2])
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(d[0]), "f"(d[1]) : "memory");
}


struct IcdSmem {
    float num[kMaxWarps][32], den[kMaxWarps][32];
    float th1[kMaxWarps][32], th2[kMaxWarps][32];
    int pos[kMaxWarps][32];
    float dx[32];
    int order[kMaxSvCols];
    int ncols, item;
};

struct IcdCount {
    unsigned long long upd, skip;
    float sum_dx, sum_x;
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
    cnt = IcdCount{};
}

// theta1 / theta2 partial sums of one lane (VEC detector rows starting at
// sinogram row offset `row0` within each A entry's row, views gfirst,
// gfirst + gstride, ... of the column): theta1 = -sum a w e,
// theta2 = sum a^2 w with a = A value x delta_t (XT_VoxUpdate.c:56-85).
template <int kUnroll, int VEC>
__device__ __forceinline__ void theta_pass(const IcdConst &K, const uint32_t *col_rec, const float *__restrict__ err,
                                           const float *__restrict__ wgt, int gfirst, int gstride, int nv, int RW,
                                           int NT, int row0, float (&th1)[VEC], float (&th2)[VEC])
{
    using VT = typename VecF<VEC>::T;
    for (int v0 = gfirst; v0 < nv; v0 += kUnroll * gstride) {
        uint4 R[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
            const int v = v0 + u * gstride;
            if (v < nv) R[u] = __ldg(reinterpret_cast<const uint4 *>(col_rec + (size_t)v * RW));
            else R[u].x = 0u;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
            const uint32_t hdr = R[u].x;
            const int cnt_q = hdr >> 24;
            // sinogram rows stay below 2^24 and N_t rows each: 32-bit offsets
            const unsigned sb = (hdr & 0xFFFFFFu) * (unsigned)NT + (unsigned)row0;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                if (q < cnt_q) {
                    float ev[VEC], wv[VEC];
                    VecF<VEC>::get(__ldcg(reinterpret_cast<const VT *>(err + (sb + (unsigned)(q * NT)))), ev);
                    VecF<VEC>::get(__ldg(reinterpret_cast<const VT *>(wgt + (sb + (unsigned)(q * NT)))), wv);
                    const float a = rec_val(R[u], q) * K.dt;
#pragma unroll
                    for (int i = 0; i < VEC; i++) {
                        float ww = wv[i];
                        if (K.huber) {
                            const float sw = sqrtf(ww);
                            if (!(fabsf(ev[i] * sw) < K.huber_T)) ww = K.huber_T * K.huber_delta * sw / fabsf(ev[i]);
                        }
                        const float aw = a * ww;
                        th2[i] += a * aw;
                        th1[i] -= ev[i] * aw;
                    }
                }
            }
        }
    }
}

// One column's theta: every lane's partial sums (theta_pass, when `run`),
// folded over the view groups of the warp and stored by group 0 into the
// warp's row of S.th1 / S.th2.
template <int kUnroll, int VEC>
__device__ __forceinline__ void theta_column(const IcdConst &K, const uint32_t *col_rec, const float *__restrict__ err,
                                             const float *__restrict__ wgt, int gfirst, int gstride, int nv, int RW,
                                             int NT, int row0, bool run, int lprp, int grp, int t0, int warp,
                                             IcdSmem &S)
{
    float th1[VEC], th2[VEC];
#pragma unroll
    for (int i = 0; i < VEC; i++) th1[i] = th2[i] = 0.0f;
    if (run) theta_pass<kUnroll, VEC>(K, col_rec, err, wgt, gfirst, gstride, nv, RW, NT, row0, th1, th2);
    for (int off = lprp; off < 32; off <<= 1) {
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            th1[i] += __shfl_xor_sync(0xffffffffu, th1[i], off);
            th2[i] += __shfl_xor_sync(0xffffffffu, th2[i], off);
        }
    }
    if (grp == 0 && run) {
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            S.th1[warp][t0 + i] = th1[i];
            S.th2[warp][t0 + i] = th2[i];
        }
    }
}

// Update the voxel columns of super-voxel (sx, sy) of frame f; the whole CTA
// cooperates (the four passes of a column are those of the one-problem sweep: neighbourhood,
// theta, solve, apply).
// kUnroll: views whose records and sinogram entries are in flight together;
// VEC: consecutive detector rows one lane owns (4 when N_t % 4 == 0, else 2);
// The data term (quadratic or generalised Huber, XT_VoxUpdate.c:68-82) is decided per
// problem at run time (K.huber).
template <int kUnroll, int VEC>
__device__ __forceinline__ void icd_update_sv(const Geom &g, const IcdLaunch &L, const IcdConst &K,
                                              const uint32_t *__restrict__ table,
                                              const int32_t *__restrict__ view_first,
                                              const uint8_t *__restrict__ mask, float *__restrict__ x,
                                              float *__restrict__ err, const float *__restrict__ wgt,
                                              float *__restrict__ mag, int f, int sx, int sy, IcdSmem &S,
                                              IcdCount &cnt)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const int NX = g.N_x, NY = g.N_y, NZ = g.N_z, NT = g.N_t, MZ = g.z_overlap;
    const int nxy = NX * NY;
    const int RW = g.rec_words;
    // A voxel column is updated in chunks of at most 32 detector rows (32 / MZ
    // voxel slices, one per lane of warp 0); chunk k covers rows [32k, 32k + 32)
    // and slices [k CZ, k CZ + CZ). Columns of up to 32 rows are one chunk.
    const int CT = NT < 32 ? NT : 32, CZ = CT / MZ;
    const int n_chunks = (NT + 31) / 32;

    // lane -> (view group, run of VEC detector rows) for the theta / apply passes
    using VT = typename VecF<VEC>::T;
    const int lpr = CT / VEC;  // lanes per sinogram row of a full chunk
    int lprp = 1;
    while (lprp < lpr) lprp <<= 1;
    const int G = 32 / lprp;  // view groups per warp
    const int grp = lane / lprp, tq = lane % lprp;
    const int t0 = tq * VEC;  // first detector row of this lane within the chunk
    const int gstride = W * G;
    const int gfirst = warp * G + grp;
    const int fv0 = view_first[f], nv = view_first[f + 1] - fv0;
    const int iter = L.iter_dev ? *L.iter_dev : L.iter;  // 1-based iteration number

    // ---- the SV's columns inside the reconstruction circle, shuffled ----------
    if (warp == 0) {
        const int ncand = L.sv * L.sv;
        int n = 0;
        for (int base = 0; base < ncand; base += 32) {
            const int i = base + lane;
            int ok = 0, c = 0;
            if (i < ncand) {
                const int j = sy * L.sv + i / L.sv, k = sx * L.sv + i % L.sv;
                if (j < NY && k < NX) {
                    c = j * NX + k;
                    ok = mask[c] && (!L.sel || L.sel[(size_t)f * nxy + c]);
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) S.order[n + __popc(m & ((1u << lane) - 1))] = c;
            n += __popc(m);
        }
        __syncwarp();
        if (lane == 0) {
            uint64_t h = mix64(L.seed ^ mix64(((uint64_t)iter << 40) ^ ((uint64_t)f << 20) ^
                                             (uint64_t)(sy * L.n_sv_x + sx)));
            for (int i = n - 1; i > 0; i--) {  // Fisher-Yates
                h = mix64(h);
                const int r = (int)(h % (uint64_t)(i + 1));
                const int t = S.order[i];
                S.order[i] = S.order[r];
                S.order[r] = t;
            }
            S.ncols = n;
        }
    }
    __syncthreads();
    const int ncols = S.ncols;
    const size_t rec_frame = (size_t)fv0 * nxy;

    for (int ci = 0; ci < ncols; ci++) {
        const int c = S.order[ci];
        const int j = c / NX, k = c - j * NX;
        const size_t col_off = ((size_t)f * nxy + c) * NZ;
        const uint32_t *col_rec = table + (rec_frame + (size_t)c * nv) * RW;

        for (int ch = 0; ch < n_chunks; ch++) {
            const int z0 = ch * CZ;                                  // first slice of the chunk
            const int cz = NZ - z0 < CZ ? NZ - z0 : CZ;              // slices in the chunk
            const int ct = cz * MZ;                                  // detector rows in the chunk
            const int rbase = ch * 32;                               // first detector row of the chunk
            const bool zl = lane < cz;
            const int z = z0 + lane;                                 // this lane's slice
            const bool row_ok = tq < ct / VEC;

            // ---- 1. neighbourhood (sources split over warps) + column activity ------
            int active_pred;
            const float V = zl ? x[col_off + z] : 0.0f;  // the column itself (warp 0 reuses it in the solve)
            {
                float num = 0.0f, den = 0.0f;
                int pos = 0;
                for (int s = warp; s < 10; s += W) {
                    if (s < 8) {
                        const int o = s < 4 ? s : s + 1;  // skip the centre of the 3x3
                        const int dy = o / 3 - 1, dx = o % 3 - 1;
                        const int jj = j + dy, kk = k + dx;
                        const bool valid = jj >= 0 && jj < NY && kk >= 0 && kk < NX;
                        const size_t noff = ((size_t)f * nxy + jj * NX + kk) * NZ;
                        const float nz0 = (valid && zl) ? x[noff + z] : 0.0f;
                        float nzm = __shfl_up_sync(0xffffffffu, nz0, 1);
                        float nzp = __shfl_down_sync(0xffffffffu, nz0, 1);
                        // across chunk edges the z +- 1 neighbours are outside the warp
                        if (lane == 0 && z > 0 && valid) nzm = x[noff + z - 1];
                        if (lane == cz - 1 && z + 1 < NZ && valid) nzp = x[noff + z + 1];
                        if (valid && zl) {
                            const float nb[3] = {nzm, nz0, nzp};
#pragma unroll
                            for (int dz = -1; dz <= 1; dz++) {
                                const int zz = z + dz;
                                if (zz < 0 || zz >= NZ) continue;
                                const float n = nb[dz + 1];
                                const float b = qg_weight(V - n, K.q, K.qmp, K.issq, K.issqp, K.cs, K.bs0);
                                const float cf = K.sf[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)] * b;
                                num += cf * n;
                                den += cf;
                                pos |= n > 0.0f;
                            }
                        }
                    } else {
                        const int ff = f + (s == 8 ? -1 : 1);
                        if (ff >= 0 && ff < g.N_time && zl) {
                            const float n = x[((size_t)ff * nxy + c) * NZ + z];
                            const float b = qg_weight(V - n, K.q, K.qmp, K.istq, K.istqp, K.ct, K.bt0);
                            const float cf = K.tf * b;
                            num += cf * n;
                            den += cf;
                            pos |= n > 0.0f;
                        }
                    }
                }
                S.num[warp][lane] = num;
                S.den[warp][lane] = den;
                S.pos[warp][lane] = pos;
                // a column is skipped only if every slice is zero with no positive
                // neighbour (in-column neighbours are the column's own values)
                active_pred = !L.zero_skipping || iter <= 1 || (zl && V != 0.0f) || pos;
            }
            // ---- 2. theta over the column's views. When the column is surely
            //         active (zero skipping off or in its first iteration, or a
            //         nonzero slice: the same test in every warp, as every warp
            //         read the column), theta runs before the barrier that also
            //         publishes the neighbourhood sums, so its loads go out without
            //         waiting for the other warps; otherwise after it, and only
            //         for an active column -------------------------------------------
            const bool sure = !L.zero_skipping || iter <= 1 || __any_sync(0xffffffffu, zl && V != 0.0f);
            if (sure)
                theta_column<kUnroll, VEC>(K, col_rec, err, wgt, gfirst, gstride, nv, RW, NT, rbase + t0, row_ok, lprp, grp,
                                           t0, warp, S);
            const int any_active = __syncthreads_or(active_pred);
            if (!any_active) {
                if (warp == 0 && zl) cnt.skip++;
                if (warp == 0 && lane == 0 && ch == 0) mag[(size_t)f * nxy + c] = 0.0f;
                continue;  // uniform across the CTA
            }
            if (!sure) {  // uniform across the CTA
                theta_column<kUnroll, VEC>(K, col_rec, err, wgt, gfirst, gstride, nv, RW, NT, rbase + t0, row_ok, lprp, grp,
                                           t0, warp, S);
                __syncthreads();
            }

            // ---- 3. zero-skipping and solve (warp 0, lane = slice of the chunk) ------
            if (warp == 0) {
                const float V0 = V;
                float numA = 0.0f, denA = 0.0f, t1 = 0.0f, t2 = 0.0f;
                int pos = 0;
                for (int w = 0; w < W; w++) {
                    numA += S.num[w][lane];
                    denA += S.den[w][lane];
                    pos |= S.pos[w][lane];
                    if (lane < ct) {
                        t1 += S.th1[w][lane];
                        t2 += S.th2[w][lane];
                    }
                }
                // in-column z - 1 / z + 1: the chunk below is already updated
                // (Gauss-Seidel over the chunks), the chunk above not yet
                const float edge_m = (z0 > 0) ? x[col_off + z0 - 1] : 0.0f;
                const float edge_p = (z0 + cz < NZ) ? x[col_off + z0 + cz] : 0.0f;
                {
                    float vm = __shfl_up_sync(0xffffffffu, V0, 1);
                    float vp = __shfl_down_sync(0xffffffffu, V0, 1);
                    if (lane == 0) vm = edge_m;
                    if (lane == cz - 1) vp = edge_p;
                    if (z >= 1 && vm > 0.0f) pos = 1;
                    if (z + 1 < NZ && vp > 0.0f) pos = 1;
                }
                const bool skip = !zl || (L.zero_skipping && iter > 1 && V0 == 0.0f && !pos);
                __syncwarp();
                S.th1[0][lane] = t1;
                S.th2[0][lane] = t2;
                __syncwarp();
                float th1 = 0.0f, th2 = 0.0f;
                if (zl)
                    for (int r = 0; r < MZ; r++) {
                        th1 += S.th1[0][lane * MZ + r];
                        th2 += S.th2[0][lane * MZ + r];
                    }
                float cur = V0;
#pragma unroll
                for (int parity = 0; parity < 2; parity++) {
                    float vm = __shfl_up_sync(0xffffffffu, cur, 1);
                    float vp = __shfl_down_sync(0xffffffffu, cur, 1);
                    if (lane == 0) vm = edge_m;
                    if (lane == cz - 1) vp = edge_p;
                    if (!skip && (z & 1) == parity) {
                        float num = numA, den = denA;
                        if (z >= 1) {
                            const float cf = K.sf[0 * 9 + 4] * qg_weight(V0 - vm, K.q, K.qmp, K.issq, K.issqp, K.cs, K.bs0);
                            num += cf * vm;
                            den += cf;
                        }
                        if (z + 1 < NZ) {
                            const float cf = K.sf[2 * 9 + 4] * qg_weight(V0 - vp, K.q, K.qmp, K.issq, K.issqp, K.cs, K.bs0);
                            num += cf * vp;
                            den += cf;
                        }
                        const float u = (num + th2 * V0 - th1) / (den + th2);
                        cur = V0 + K.alpha * (u - V0);
                    }
                }
                const float dx = skip ? 0.0f : cur - V0;
                S.dx[lane] = dx;
                if (zl) {
                    if (!skip) {
                        x[col_off + z] = cur;
                        cnt.upd++;
                        cnt.sum_dx += fabsf(dx);
                        cnt.sum_x += fabsf(cur);
                    } else {
                        cnt.skip++;
                    }
                }
                float m = fabsf(dx);
                for (int off = 16; off > 0; off >>= 1) m += __shfl_xor_sync(0xffffffffu, m, off);
                if (lane == 0) {
                    float *mp = mag + (size_t)f * nxy + c;
                    *mp = ch == 0 ? m : *mp + m;
                }
            }
            __syncthreads();

            // ---- 4. apply e -= a dx (the next chunk's or column's barrier orders
            //         these reductions before its theta loads) ---------------------------
            {
                float dxv[VEC];
                bool any = false;
#pragma unroll
                for (int i = 0; i < VEC; i++) {
                    dxv[i] = row_ok ? S.dx[(t0 + i) / MZ] : 0.0f;
                    any |= dxv[i] != 0.0f;
                }
                if (any) {
                    for (int v0 = gfirst; v0 < nv; v0 += kUnroll * gstride) {
                        uint4 R[kUnroll];
#pragma unroll
                        for (int u = 0; u < kUnroll; u++) {
                            const int v = v0 + u * gstride;
                            if (v < nv) R[u] = __ldg(reinterpret_cast<const uint4 *>(col_rec + (size_t)v * RW));
                            else R[u].x = 0u;
                        }
#pragma unroll
                        for (int u = 0; u < kUnroll; u++) {
                            const uint32_t hdr = R[u].x;
                            const int cnt_q = hdr >> 24;
                            const unsigned sb = (hdr & 0xFFFFFFu) * (unsigned)NT + (unsigned)(rbase + t0);
#pragma unroll
                            for (int q = 0; q < 3; q++) {
                                if (q < cnt_q) {
                                    const float a = -(rec_val(R[u], q) * K.dt);
                                    float d[VEC];
#pragma unroll
                                    for (int i = 0; i < VEC; i++) d[i] = a * dxv[i];
                                    red_add(err + (sb + (unsigned)(q * NT)), d);
                                }
                            }
                        }
                    }
                }
            }
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Many independent problems in one persistent launch per colour phase. The
// queue runs over the SV items of every problem of the launch, interleaved in
// proportion to each problem's item count (item_map[] gives the problem and
// its item), so the CTAs working at any moment spread over the problems; a
// CTA keeps the descriptor of its current problem in shared memory and
// reloads it when its next item belongs to another problem. Problems of one
// launch share the detector-row vector width (a template parameter).
template <int kUnroll, int VEC>
__global__ void __launch_bounds__(kMaxWarps * 32, 4) icd_batch_kernel(const BatchDesc *__restrict__ descs,
                                                                      const int2 *__restrict__ item_map, int total,
                                                                      int phase, unsigned int *__restrict__ queue)
{
    __shared__ IcdSmem S;
    __shared__ __align__(16) BatchDesc P;
    int cur = -1;
    IcdCount cnt{};
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) S.item = (int)atomicAdd(queue, 1u);
        __syncthreads();
        const int item = S.item;
        if (item >= total) break;
        const int2 pm = item_map[item];  // (problem, item of that problem)
        if (pm.x != cur) {                // uniform
            if (cur >= 0) flush_counts(cnt, P.stats);
            __syncthreads();
            const int4 *src = reinterpret_cast<const int4 *>(descs + pm.x);
            int4 *dst = reinterpret_cast<int4 *>(&P);
            for (int i = threadIdx.x; i < (int)(sizeof(BatchDesc) / sizeof(int4)); i += blockDim.x) dst[i] = src[i];
            __syncthreads();
            cur = pm.x;
        }
        if (!P.active) continue;
        const int K = P.L.colors_k;
        const int hx = (P.L.n_sv_x + K - 1) / K, slots = hx * ((P.L.n_sv_y + K - 1) / K);
        const int f = pm.y % P.g.N_time;
        const int rem = (int)((long long)(pm.y / P.g.N_time) * P.L.perm % slots);
        const int color = (phase + f) % (K * K);
        const int sx = K * (rem % hx) + color % K;
        const int sy = K * (rem / hx) + color / K;
        if (sx >= P.L.n_sv_x || sy >= P.L.n_sv_y) continue;
        icd_update_sv<kUnroll, VEC>(P.g, P.L, P.K, P.table, P.view_first, P.mask, P.x, P.err, P.w, P.mag, f, sx, sy, S,
                                    cnt);
    }
    if (cur >= 0) flush_counts(cnt, P.stats);
}

// Before an iteration: advance every problem's iteration number and clear its counters.
__global__ void batch_begin_iteration(BatchDesc *descs, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    descs[i].L.iter += 1;
    *descs[i].stats = IcdStats{};
}

// After an iteration: accumulate the updates and stop problems whose
// convergence statistic 100 sum|dx| / sum|x| fell below their threshold after
// the first iteration (XT_ICD_update.c:1083-1090).
__global__ void batch_end_iteration(BatchDesc *descs, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !descs[i].active) return;
    const IcdStats s = *descs[i].stats;
    descs[i].total_updates += s.updates;
    descs[i].iters_done = descs[i].L.iter;
    const double pct = s.sum_abs_x > 0 ? 100.0 * s.sum_abs_dx / s.sum_abs_x : 0.0;
    descs[i].last_pct = pct;
    if (descs[i].L.iter > 1 && pct < descs[i].convg_thresh) descs[i].active = 0;
}

int batch_grid(int vec, int warps)
{
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (vec == 4) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, icd_batch_kernel<2, 4>, warps * 32, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, icd_batch_kernel<2, 2>, warps * 32, 0);
    return sms * (per_sm > 0 ? per_sm : 1);
}

void launch_icd_batch(int vec, int warps, int grid, const BatchDesc *d_descs, const int2 *d_item_map, int total,
                      int phase, unsigned int *d_queue, cudaStream_t st)
{
    if (vec == 4) icd_batch_kernel<2, 4><<<grid, warps * 32, 0, st>>>(d_descs, d_item_map, total, phase, d_queue);
    else icd_batch_kernel<2, 2><<<grid, warps * 32, 0, st>>>(d_descs, d_item_map, total, phase, d_queue);
}

void launch_batch_begin(BatchDesc *d_descs, int n, cudaStream_t st)
{
    batch_begin_iteration<<<(n + 127) / 128, 128, 0, st>>>(d_descs, n);
}

void launch_batch_end(BatchDesc *d_descs, int n, cudaStream_t st)
{
    batch_end_iteration<<<(n + 127) / 128, 128, 0, st>>>(d_descs, n);
}

}  // namespace mbirgpu
