"""The cost kernel's prior term over its range of differences, against the oracle in FP64.

Cases: zero differences, differences down to FP32's subnormals and up to 1e30
(where the denominator leaves the fast form's range), few slices and
more slices than a warp has lanes, several frames, each form of q.

Tolerance: a term is off by a few 2^-50 (the truncated series, the cubic step of
the reciprocal) and the oracle's sum of N <= 4e5 positive terms by up to
N 2^-53 = 4.4e-11; 5e-11 holds both.
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow,nframe,p,quad,span", [
    (24, 6, 2, 1.2, 1, (0, 0)),      # ordinary differences
    (24, 6, 2, 1.2, 0, (0, 0)),
    (20, 40, 1, 1.1, 1, (-38, 0)),   # 40 slices; subnormal differences
    (20, 40, 1, 1.3, 0, (-38, 0)),
    (16, 8, 3, 2.0, 1, (-20, 2)),
    (16, 4, 3, 1.2, 1, (0, 30)),     # denominators past 2^100
    (16, 4, 1, 1.2, 0, (-44, 30)),
    (8, 16, 1, 1.2, 1, None),        # all zero
])
def test_prior_term_over_the_range_of_differences(ncol, nrow, nframe, p, quad, span):
    pb, obj = make_problem(ncol=ncol, nrow=nrow, nview=12 * nframe, nframe=nframe, p=p, seed=3, quad_convex=quad)
    rng = np.random.default_rng(5)
    if span is None:
        x = np.zeros(obj.shape, np.float32)
    else:
        e = rng.integers(span[0], span[1] + 1, size=obj.shape)
        x = (rng.normal(size=obj.shape) * 10.0**e * (rng.random(obj.shape) < 0.7)).astype(np.float32)
    opt = pc.get_options()
    opt.mrf_p = p  # the options carry the potential's p
    s = pc.Session(to_gpu_problem(pb), options=opt)
    s.set_object(x)
    prior = s.cost()[2]
    ref = O.Oracle(pb).cost(np.zeros(s.get_error().shape, np.float32), x)[2]
    if span is None:
        assert prior == ref == 0
    else:
        assert np.isfinite(ref) and prior == pytest.approx(ref, rel=5e-11)
