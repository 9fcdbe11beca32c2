"""ICD with q < 2, or q = p, where voxels differ by less than the smallest normal FP32
number: the hardware logarithm takes such a difference for zero, so the surrogate weight
at zero stands for it, inside the volume and against its border. Two iterations from an
object of such values leave it finite and lower its cost (a surrogate step never raises
it; one super-voxel, so the columns are updated one after another).
"""
import numpy as np
import pytest

import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrow,nframe,p,q", [(8, 1, 1.1, 1.9), (6, 2, 1.2, 1.5), (8, 1, 1.5, 1.5), (8, 1, 2.0, 2.0)])
def test_differences_below_the_normal_range_count_as_none(nrow, nframe, p, q):
    pb, obj = make_problem(ncol=16, nrow=nrow, nview=20 * nframe, nframe=nframe, seed=3)
    rng = np.random.default_rng(2)
    tiny = np.where(rng.random(obj.shape) < 0.5, 1e-40, -3e-39).astype(np.float32)
    keep = rng.random(obj.shape) < 0.4
    o = pc.get_options()
    o.mrf_p, o.mrf_q, o.sv_size, o.sv_colors, o.cta_warps, o.zero_skipping, o.nhicd_passes = p, q, 16, 2, 4, 0, 0
    s = pc.Session(to_gpu_problem(pb), options=o)
    s.set_object(np.where(keep, obj, tiny).astype(np.float32))
    before = s.cost()[0]
    for it in (1, 2):
        s.icd_iteration(it)
        assert np.isfinite(s.get_object()).all() and np.isfinite(s.get_error()).all()
        after = s.cost()[0]
        assert after < before
        before = after
    s.close()
