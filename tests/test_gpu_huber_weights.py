"""The sweep's generalised-Huber weights over their range, against the sequential FP64
restatement of test_gpu_icd_sweep.py (one super-voxel; tolerance derived there: the
weights' rounding, 4 2^-24, is below the theta sums').

Cases: all entries linear (from zero), few (from the true object), thresholds and delta
where the short form of the linear weight does not hold (zero, tiny, large), small weights
and outliers beyond its range, both widths of a lane's rows, four and eight entries in flight.
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem
from test_gpu_icd_sweep import sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrow,T,delta,start,wscale,outlier,opts", [
    (8, 4.0, 0.5, "zero", 1.0, 2.0, {}),
    (8, 4.0, 0.5, "true", 1.0, 2.0, {}),
    (6, 3.7, 0.31, "zero", 1.0, 2.0, {}),
    (6, 3.7, 0.31, "true", 1.0, 2.0, dict(icd_unroll=1)),
    (8, 0.5, 1.0, "true", 1.0, 0.0, dict(icd_unroll=1)),
    (8, 0.0, 0.5, "true", 1.0, 0.0, {}),
    (8, 4.0, 0.0, "true", 1.0, 0.0, {}),
    (8, 1e-6, 0.3, "true", 1.0, 0.0, {}),
    (8, 1e-25, 0.3, "true", 1.0, 0.0, {}),
    (8, 1e6, 0.5, "true", 1.0, 0.0, {}),
    (8, 4.0, 0.5, "true", 1e-17, 0.0, {}),
    (8, 4.0, 0.5, "true", 1.0, 1e18, {}),
    (8, 1e18, 1e-18, "true", 1.0, 1e18, {}),
])
def test_linear_weights_match_fp64_updates(nrow, T, delta, start, wscale, outlier, opts):
    pb, obj = make_problem(ncol=16, nrow=nrow, nview=20, seed=3, quad_convex=0, huber_T=T, huber_delta=delta)
    pb.projections[::3, ::2, ::5] += outlier
    pb.weights *= np.float32(wscale)
    orc = O.Oracle(pb)
    o = pc.get_options()
    o.mrf_p, o.sv_size, o.sv_colors, o.nhicd_passes, o.refresh_every, o.cta_warps = pb.mrf_p, 16, 2, 0, 0, 4
    for k, v in opts.items():
        setattr(o, k, v)
    s = pc.Session(to_gpu_problem(pb), options=o)
    first, count, vals = s.amatrix()
    A = [[(int(first[v].flat[c]), vals[v].reshape(-1, vals.shape[-1])[c, :count[v].flat[c]].astype(np.float64))
          for c in range(first[v].size)] for v in range(20)]
    x = obj.astype(np.float64) if start == "true" else np.zeros(orc.shape)
    s.set_object(x.astype(np.float32))
    e, w = s.get_error().astype(np.float64), orc.w.astype(np.float64)
    for it in (1, 2):
        s.icd_iteration(it)
        sweep(orc, [range(20)], A, x, e, w, it, 16, int(o.seed), True)
        got = s.get_object()
        assert np.isfinite(got).all()
        assert np.abs(got - x).max() <= 1e-3 * np.abs(x).max(), (it, np.abs(got - x).max(), np.abs(x).max())
        assert np.abs(s.get_error() - e).max() <= 1e-3 * np.abs(orc.y).max(), it
    s.close()
