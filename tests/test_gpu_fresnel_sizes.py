"""The Fresnel passes where their forms meet: 256-point sequences along rows, columns or
both, twiddle tables longer than the sequence, the smallest and largest lengths, every
radix of the generic stages.

Tolerance: forward and inverse transform of R C points, each stage's rounding at most
2 2^-24 of a value, log2(R C) stages twice, and 1.5 for the transfer factor and the
spread of the values: 6 log2(R C) 2^-24 of the largest (6.4e-6 for 2^18 points).
"""
import numpy as np
import pytest

from test_gpu_pc import P, scan
from phasecon_b200.pcmbir import PcSession, default_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,C,radix", [
    (256, 256, 16), (256, 16, 16), (16, 256, 16), (256, 1024, 16), (1024, 256, 16), (512, 256, 16),
    (64, 512, 16), (4, 1024, 16), (1024, 4, 16), (32, 128, 8), (128, 32, 4), (64, 256, 2), (256, 256, 4),
])
def test_transform_matches_fp64(R, C, radix):
    V = 2
    pb, g, _, _, _ = scan(V, R, C, seed=3)
    s = PcSession(pb, default_options(fft_radix=radix))
    rng = np.random.default_rng(1)
    x = (rng.normal(size=(V, R, C)) + 1j * rng.normal(size=(V, R, C))).astype(np.complex64)
    tol = 6 * np.log2(R * C) * 2.0**-24
    for herm in (False, True):
        out = s.fresnel(x, herm)
        for v in range(V):
            ref = P.fresnel(g, x[v].astype(np.complex128), herm)
            assert np.abs(out[v] - ref).max() <= tol * np.abs(ref).max()
    s.close()
