"""The ICD sweep's neighbourhood tile where super-voxels border on each other, against the
sequential FP64 restatement of test_gpu_icd_sweep.py (tolerance derived there).

The image is two by two super-voxels of four colours: each colour phase updates one
super-voxel a frame, so the order is fixed, and between them the four have every side and
corner of the tile inside the image.

Cases: tiles brought by bulk copies (slices a multiple of 4) and by plain loads, one and
two chunks of rows, a tile clipped by the image, one and three frames, coarse voxel
scales, the Huber data term, several widths of a CTA, records not staged (no tile).
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem
from test_gpu_icd_sweep import sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow,nview,nframe,scale,huber,opts", [
    (8, 8, 20, 1, (1, 1), 0, dict(cta_warps=4)),
    (8, 8, 12, 3, (1, 1), 0, dict(cta_warps=2)),
    (8, 6, 20, 1, (1, 1), 0, dict(cta_warps=4)),
    (8, 6, 14, 3, (1, 1), 1, dict(cta_warps=8)),
    (6, 8, 20, 3, (1, 1), 0, dict(cta_warps=2)),
    (8, 32, 16, 3, (1, 1), 0, dict(cta_warps=2)),
    (8, 32, 16, 1, (1, 1), 1, dict(cta_warps=1)),
    (8, 38, 16, 1, (1, 1), 1, dict(cta_warps=8)),
    (8, 38, 12, 3, (1, 1), 0, dict(cta_warps=4)),
    (8, 64, 12, 3, (1, 1), 0, dict(cta_warps=4)),
    (8, 64, 12, 1, (1, 1), 1, dict(cta_warps=2)),
    (8, 64, 12, 1, (1, 2), 0, dict(cta_warps=4)),
    (16, 16, 16, 2, (2, 2), 0, dict(cta_warps=4)),
    (8, 8, 12, 3, (1, 1), 1, dict(cta_warps=4, stage_records=0)),
])
def test_super_voxels_read_their_neighbours(ncol, nrow, nview, nframe, scale, huber, opts):
    pb, _ = make_problem(ncol=ncol, nrow=nrow, nview=nview * nframe, nframe=nframe, seed=4, sig_t=0.01,
                         quad_convex=0 if huber else 1, moving=True)
    if huber:
        pb.projections[::3, ::2, ::5] += 2.0
    orc = O.Oracle(pb, *scale)
    o = pc.get_options()
    o.mrf_p, o.sv_size, o.sv_colors, o.nhicd_passes, o.refresh_every = pb.mrf_p, 4, 2, 0, 0
    for k, v in opts.items():
        setattr(o, k, v)
    s = pc.Session(to_gpu_problem(pb), *scale, options=o)
    first, count, vals = s.amatrix()
    V = nview * nframe
    A = [[(int(first[v].flat[c]), vals[v].reshape(-1, vals.shape[-1])[c, :count[v].flat[c]].astype(np.float64))
          for c in range(first[v].size)] for v in range(V)]
    edges = pb.recon_times
    frames_views = [[v for v in range(V) if edges[f] <= pb.proj_times[v] < edges[f + 1]] for f in range(nframe)]
    s.set_object_zero()
    x, e = np.zeros(orc.shape), orc.y.astype(np.float64)
    w = orc.w.astype(np.float64)
    for it in (1, 2, 3):
        st = s.icd_iteration(it)
        sweep(orc, frames_views, A, x, e, w, it, 4, int(o.seed), bool(huber))
        assert st.voxel_updates > 0
        got = s.get_object()
        assert np.abs(got - x).max() <= 1e-3 * np.abs(x).max(), (it, np.abs(got - x).max(), np.abs(x).max())
        assert np.abs(s.get_error() - e).max() <= 1e-3 * np.abs(orc.y).max(), it
    s.close()


@pytest.mark.parametrize("nrow,huber,warps", [(8, 0, 4), (6, 0, 2), (32, 1, 4), (38, 0, 8), (64, 1, 1)])
def test_one_cta_refills_its_tile(nrow, huber, warps):
    """2 x 2 super-voxels on a 14 x 14 image: one CTA (the bound on columns in flight) takes
    all of a colour in turn. With and without tile it makes the same updates in the same
    order, so both are within the restatement's bound of the same image."""
    pb, _ = make_problem(ncol=14, nrow=nrow, nview=20, nframe=1, seed=4, quad_convex=0 if huber else 1)
    images = []
    for staged in (1, 0):
        o = pc.get_options()
        o.mrf_p, o.sv_size, o.sv_colors, o.nhicd_passes, o.refresh_every = pb.mrf_p, 2, 2, 0, 0
        o.cta_warps, o.stage_records = warps, staged
        s = pc.Session(to_gpu_problem(pb), options=o)
        s.set_object_zero()
        for it in (1, 2, 3):
            s.icd_iteration(it)
        images.append((s.get_object(), s.get_error()))
        s.close()
    for a, b in zip(*images):
        assert np.abs(b).max() > 0 and np.abs(a - b).max() <= 2e-3 * np.abs(b).max()
