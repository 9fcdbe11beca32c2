"""The ICD sweep on columns of more than 32 detector rows whose slices' rows do not divide
32, against the sequential FP64 restatement of test_gpu_icd_sweep.py (one super-voxel, so
the order is fixed; tolerance derived there).

Cases: chunks of rows that start on odd rows, slices across a multiple of 32 rows, a last
chunk of fewer slices, slices of 17 to 31 rows (one a chunk) and of more than 32 (several
blocks of rows), row counts that are multiples of 4 and not, lists of one and of several
blocks of views, coarse columns, several frames, the Huber data term, every width of a CTA.
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem
from test_gpu_icd_sweep import sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow,nview,nframe,scale,huber,warps", [
    (16, 42, 18, 1, (1, 3), 0, 4),
    (16, 96, 12, 2, (1, 3), 1, 8),
    (16, 36, 15, 1, (1, 9), 0, 2),
    (16, 40, 15, 1, (1, 5), 1, 1),
    (16, 34, 14, 1, (1, 17), 0, 4),
    (16, 62, 9, 1, (1, 31), 0, 4),
    (16, 96, 9, 2, (1, 48), 0, 4),
    (16, 66, 9, 1, (1, 33), 1, 2),
    (16, 130, 7, 1, (1, 65), 0, 8),
    (16, 64, 9, 1, (1, 64), 0, 4),
    (16, 42, 400, 1, (1, 6), 0, 1),
    (16, 66, 300, 1, (1, 33), 0, 1),
    (32, 36, 12, 1, (2, 6), 1, 2),
    (64, 42, 8, 1, (4, 7), 0, 4),
])
def test_sweep_over_z_scales(ncol, nrow, nview, nframe, scale, huber, warps):
    pb, _ = make_problem(ncol=ncol, nrow=nrow, nview=nview, nframe=nframe, seed=3, sig_t=0.01,
                         quad_convex=0 if huber else 1, moving=True)
    if huber:
        pb.projections[::3, ::2, ::5] += 2.0
    orc = O.Oracle(pb, *scale)
    o = pc.get_options()
    o.mrf_p, o.sv_size, o.sv_colors, o.nhicd_passes, o.refresh_every, o.cta_warps = pb.mrf_p, 16, 2, 0, 0, warps
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
        assert np.abs(s.get_error() - e).max() <= 1e-3 * np.abs(orc.y).max(), it
    s.close()
