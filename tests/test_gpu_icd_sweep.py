"""The ICD sweep against a sequential FP64 restatement of the same updates.

A 16 x 16 image is one super-voxel (sv_size 16), so its columns are updated one
after another in the kernel's seeded order and the result does not depend on
timing: two iterations (the first without zero skipping, the second with it)
are repeated here in FP64 -- theta over the column's A entries
(MBIR_4D/XT_VoxUpdate.c:45-117), even slices then odd ones through the
oracle's surrogate weights (XT_ICD_update.c:133-182), e updated per column.

Cases: every layout of a column over the warps, records staged or unpacked in
blocks of views, slabs of more than 32 rows, rows and slices that are not
multiples of 4, coarse voxel scales, several frames, the Huber data term.

Tolerance: a theta sum of N <= 700 FP32 terms is off by up to N 2^-24 of its
terms' sum and a surrogate weight by a few 2^-22, 5e-5 together; the coupled
updates of 2 x 208 columns leave that below 1e-3 of the largest value.
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def sv_order(n, seed, it, f, sv_index):
    """The kernel's shuffle of an SV's n columns (row-major inside the SV)."""
    order = list(range(n))
    h = mix64(seed ^ mix64((it << 40) ^ (f << 20) ^ sv_index))
    for i in range(n - 1, 0, -1):
        h = mix64(h)
        r = h % (i + 1)
        order[i], order[r] = order[r], order[i]
    return order


def sweep(orc, frames_views, A, x, e, w, it, sv, seed, huber):
    """One full sweep, super-voxel by super-voxel, in FP64 (x [T][Z][Y][X], e [view][col][row])."""
    g = orc.g
    NZ, NY, NX, MZ = g.N_z, g.N_y, g.N_x, g.z_overlap
    mask = orc.mask()
    nsx = (NX + sv - 1) // sv
    sf = np.array(g.spatial_filter).reshape(3, 3, 3)

    def coef(d, f, sq, sqp, c):
        ad = np.abs(d)
        with np.errstate(divide="ignore", invalid="ignore"):
            t1 = ad ** (g.q - g.p) / sqp
            b = ad ** (g.q - 2) * (g.q - (g.q - g.p) * t1 / (c + t1)) / ((c + t1) * sq)
        return f * np.where(d == 0, g.q / (sq * c), b)

    for phase in range(4):
        for f in range(g.N_time):
            color = (phase + f) % 4
            for sy in range(color // 2, (NY + sv - 1) // sv, 2):
                for sx in range(color % 2, nsx, 2):
                    cols = [(j, k) for j in range(sy * sv, min(sy * sv + sv, NY)) for k in
                            range(sx * sv, min(sx * sv + sv, NX)) if mask[j, k]]
                    for o in sv_order(len(cols), seed, it, f, sy * nsx + sx):
                        j, k = cols[o]
                        cz_all = max(1, min(32, g.N_t) // MZ)
                        for z0 in range(0, NZ, cz_all):
                            zs = np.arange(z0, min(z0 + cz_all, NZ))
                            V = x[f, zs, j, k].copy()
                            num, den, pos = np.zeros(len(zs)), np.zeros(len(zs)), np.zeros(len(zs), bool)
                            for dy in (-1, 0, 1):
                                for dx in (-1, 0, 1):
                                    if (dy or dx) and 0 <= j + dy < NY and 0 <= k + dx < NX:
                                        for dz in (-1, 0, 1):
                                            ok = (zs + dz >= 0) & (zs + dz < NZ)
                                            n = np.where(ok, x[f, np.clip(zs + dz, 0, NZ - 1), j + dy, k + dx], 0)
                                            c = np.where(ok, coef(V - n, sf[dz + 1, dy + 1, dx + 1], g.sigma_s_q,
                                                                  g.sigma_s_q_p, g.c_s), 0)
                                            num, den, pos = num + c * n, den + c, pos | (ok & (n > 0))
                            for ff in (f - 1, f + 1):
                                if 0 <= ff < g.N_time:
                                    n = x[ff, zs, j, k]
                                    c = coef(V - n, g.time_filter, g.sigma_t_q, g.sigma_t_q_p, g.c_t)
                                    num, den, pos = num + c * n, den + c, pos | (n > 0)
                            below = x[f, np.maximum(zs - 1, 0), j, k] * (zs > 0)
                            above = x[f, np.minimum(zs + 1, NZ - 1), j, k] * (zs + 1 < NZ)
                            if it > 1 and not (V != 0).any() and not pos.any():
                                continue
                            rows = slice(z0 * MZ, (zs[-1] + 1) * MZ)
                            t1, t2 = np.zeros(len(zs) * MZ), np.zeros(len(zs) * MZ)
                            for v in frames_views[f]:
                                first, vals = A[v][j * NX + k]
                                for q, a in enumerate(vals):
                                    a = a * g.delta_t
                                    ee, ww = e[v, first + q, rows], w[v, first + q, rows]
                                    if huber:
                                        s = np.sqrt(ww)
                                        ww = np.where(np.abs(ee * s) < g.huber_T, ww, g.huber_T * g.huber_delta * s /
                                                      np.maximum(np.abs(ee), 1e-300))
                                    t1 -= a * ww * ee
                                    t2 += a * a * ww
                            t1, t2 = t1.reshape(-1, MZ).sum(1), t2.reshape(-1, MZ).sum(1)
                            skip = (it > 1) & (V == 0) & ~(pos | (below > 0) | (above > 0))
                            cur = V.copy()
                            for parity in (0, 1):
                                vm = np.concatenate([[below[0]], cur[:-1]])
                                vp = np.concatenate([cur[1:], [above[-1]]])
                                cm = np.where(zs > 0, coef(V - vm, sf[0, 1, 1], g.sigma_s_q, g.sigma_s_q_p, g.c_s), 0)
                                cp = np.where(zs + 1 < NZ, coef(V - vp, sf[2, 1, 1], g.sigma_s_q, g.sigma_s_q_p, g.c_s), 0)
                                u = (num + cm * vm + cp * vp + t2 * V - t1) / (den + cm + cp + t2)
                                go = (zs % 2 == parity) & ~skip
                                cur = np.where(go, V + g.alpha * (u - V), cur)
                            x[f, zs, j, k] = cur
                            d = np.repeat(cur - V, MZ)
                            for v in frames_views[f]:
                                first, vals = A[v][j * NX + k]
                                for q, a in enumerate(vals):
                                    e[v, first + q, rows] -= a * g.delta_t * d


CASES = [
    # ncol, nrow, views, frames, scale (xy, z), Huber, options
    (16, 8, 20, 1, (1, 1), 0, dict(cta_warps=4)),
    (16, 8, 20, 1, (1, 1), 0, dict(cta_warps=1)),
    (16, 6, 21, 2, (1, 1), 0, dict(cta_warps=8)),                    # 2-row lanes, slices not a multiple of 4
    (16, 32, 19, 1, (1, 1), 1, dict(cta_warps=2, icd_unroll=1)),
    (16, 38, 18, 1, (1, 1), 1, dict(cta_warps=8)),                   # two chunks of rows
    (16, 64, 9, 1, (1, 1), 0, dict(cta_warps=4, icd_unroll=2)),
    (32, 16, 20, 1, (2, 2), 0, dict(cta_warps=4)),                   # coarse scales
    (64, 12, 16, 1, (4, 1), 0, dict(cta_warps=4)),
    (32, 36, 12, 1, (2, 2), 1, dict(cta_warps=2)),
    (16, 8, 20, 1, (1, 1), 0, dict(cta_warps=4, stage_records=0)),   # lists unpacked where they are used
    (16, 38, 18, 2, (1, 1), 1, dict(cta_warps=2, stage_records=0)),
    (16, 32, 700, 1, (1, 1), 0, dict(cta_warps=1, stage_records=0)),  # ... in several blocks of views
    (16, 4, 700, 1, (1, 1), 0, dict(cta_warps=8)),
]


@pytest.mark.parametrize("ncol,nrow,nview,nframe,scale,huber,opts", CASES)
def test_sweep_matches_sequential_fp64_updates(ncol, nrow, nview, nframe, scale, huber, opts):
    pb, _ = make_problem(ncol=ncol, nrow=nrow, nview=nview, nframe=nframe, seed=3, sig_t=0.01,
                         quad_convex=0 if huber else 1, moving=True)
    if huber:  # zingers: entries on the linear branch
        pb.projections[::3, ::2, ::5] += 2.0
    orc = O.Oracle(pb, *scale)
    o = pc.get_options()
    o.mrf_p, o.sv_size, o.sv_colors, o.nhicd_passes, o.refresh_every = pb.mrf_p, 16, 2, 0, 0
    for k, v in opts.items():
        setattr(o, k, v)
    s = pc.Session(to_gpu_problem(pb), *scale, options=o)
    first, count, vals = s.amatrix()
    A = [[(int(first[v].flat[c]), vals[v].reshape(-1, vals.shape[-1])[c, :count[v].flat[c]].astype(np.float64))
          for c in range(first[v].size)] for v in range(nview)]
    edges = pb.recon_times
    frames_views = [[v for v in range(nview) if edges[f] <= pb.proj_times[v] < edges[f + 1]] for f in range(nframe)]
    s.set_object_zero()
    x, e = np.zeros(orc.shape), orc.y.astype(np.float64)
    w = orc.w.astype(np.float64)
    for it in (1, 2):
        st = s.icd_iteration(it)
        sweep(orc, frames_views, A, x, e, w, it, 16, int(o.seed), bool(huber))
        assert st.voxel_updates > 0
        got = s.get_object()
        assert np.isfinite(got).all()
        assert np.abs(got - x).max() <= 1e-3 * np.abs(x).max(), (it, np.abs(got - x).max(), np.abs(x).max())
        err = s.get_error()
        assert np.abs(err - e).max() <= 1e-3 * np.abs(orc.y).max(), it
    s.close()
