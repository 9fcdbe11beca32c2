"""The proximal sweep's packed cost in its two forms (q - p above zero, and not) where
they could differ: equal neighbours, whose differences are zero, in every
lanes-per-pixel layout.

One sweep against the oracle's raster order; the bound is the one of
test_nelder_mead_sweep_matches_oracle (median 3e-4, largest 1e-2 of the range), which
covers searches that stop a step apart.
"""
import numpy as np
import pytest

from test_gpu_pc import P, gpu_nms_sweep, nms_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("p", [1.2, 2.0])
def test_sweep_from_equal_neighbours_matches_oracle(lanes, p):
    pb, g, zr0, zi0, w0, om0, vd = nms_case(1, 32, 16, seed=5)
    g.mrf_p = p
    zr0, zi0 = np.full_like(zr0, 0.02), np.full_like(zi0, 0.1)
    zr1, zi1 = gpu_nms_sweep(pb, zr0, zi0, w0, om0, vd, nms_order=0, nms_lanes=lanes, nms_ctas_per_view=2, mrf_p=p)
    ar, ai = zr0[0].copy(), zi0[0].copy()
    P.nms_sweep(g, ar, ai, w0[0] - vd[0].astype(np.complex128), order="raster")
    for got, ref in ((zr1[0], ar), (zi1[0], ai)):
        d = np.abs(got - ref) / np.abs(ref).max()
        assert np.median(d) <= 3e-4 and d.max() <= 1e-2
